// FP32 CSR SpMM for sm_100a: C = A * B with A in CSR, B and C dense row-major.
//
// Replaces the reference's GESpMM / LBSpMM kernel set (spmm/mm/spmm_kernel.cu:247-477).
// Scheduling: the nnz axis is cut into chunks of a nominal size S.  A cut that falls
// inside a row no longer than S is moved back to the start of that row, so short rows
// stay whole; a cut inside a longer ("heavy") row stays where it is, so heavy rows are
// split across chunks (a merge-path split restricted to heavy rows).  One warp owns one
// chunk; the kernel is in spmm_warp.cuh, its instances per vector width in spmm_shapes_v*.cu,
// the tables it walks are built in structure_kernels.cu.  This file holds the entry points, the
// choice of chunk size and shape, the row-split kernels and the TMA-fed kernel.
// HPSPMM_ALGO_ROW_SPLIT keeps the reference's GESpMM shape (one sub-warp per row, every row
// summed in storage order), which reproduces the CPU oracle bit for bit.
#include <algorithm>
#include <mutex>
#include <new>

#include <cuda.h>   // CUtensorMap and the encode prototype; the entry point is looked up at run time

#include "device_utils.cuh"
#include "hpspmm_internal.h"
#include "spmm_warp.cuh"

namespace {

using namespace hpspmm;

constexpr int kBlockThreads = 256;

// ---- row-split kernel: one W-lane worker per row, K = 4 * W * R --------------------------------
// HPSPMM_ALGO_ROW_SPLIT: the shape of the reference's GESpMM, every row summed in storage order.
template <int W, int R, int U, int MINB, bool HINT>
__global__ void __launch_bounds__(kBlockThreads, MINB)
spmm_rowsplit_kernel(int M, const int* __restrict__ row_ptr, const int* __restrict__ col_idx,
                     const float* __restrict__ vals, const float* __restrict__ B, float* __restrict__ C) {
  constexpr int K = 4 * W * R;
  constexpr int T = 32;       // entries per staged (col, val) tile
  constexpr int RT = T / W;   // entries each lane stages per tile
  constexpr int STAGES = 2;
  __shared__ int2 tiles[kBlockThreads / W][STAGES][T];

  const int lane = threadIdx.x & (W - 1);
  const int row = (int)(((int64_t)blockIdx.x * kBlockThreads + threadIdx.x) / W);
  if (row >= M) return;
  const unsigned mask = subwarp_mask<W>();
  const uint64_t policy = HINT ? policy_evict_last() : 0ull;
  int2(*my)[T] = tiles[threadIdx.x / W];
  const int n0 = __ldg(row_ptr + row);
  const int n1 = __ldg(row_ptr + row + 1);

  // (col, val) pairs travel global -> shared with 4-byte asynchronous copies, two tiles
  // ahead of their use; entries past the end of the row are staged as (column 0, 0.0f).
  auto stage_tile = [&](int stage, int base) {
#pragma unroll
    for (int t = 0; t < RT; ++t) {
      const int e = t * W + lane;
      const int j = base + e;
      if (j < n1) {
        cp_async_4(&my[stage][e].x, col_idx + j);
        cp_async_4(&my[stage][e].y, vals + j);
      } else {
        my[stage][e] = make_int2(0, 0);
      }
    }
    cp_async_commit();
  };
  stage_tile(0, n0);
  stage_tile(1, n0 + T);

  float4 acc[R];
#pragma unroll
  for (int r = 0; r < R; ++r) acc[r] = make_float4(0.f, 0.f, 0.f, 0.f);
  const float* Bl = B + lane * 4;

  int stage = 0;
  for (int base = n0; base < n1; base += T) {
    cp_async_wait<STAGES - 1>();
    __syncwarp(mask);
#pragma unroll 1
    for (int u0 = 0; u0 < T; u0 += U) {
      const int j0 = base + u0;
      if (j0 >= n1) break;
      float4 b[U][R];
      float v[U];
#pragma unroll
      for (int i = 0; i < U; ++i) {
        const int2 e = my[stage][u0 + i];  // same address for the whole worker: a broadcast
        v[i] = __int_as_float(e.y);
        const float* p = Bl + (int64_t)e.x * K;
#pragma unroll
        for (int r = 0; r < R; ++r) b[i][r] = ld_gather<HINT>(p + r * W * 4, policy);
      }
#pragma unroll
      for (int i = 0; i < U; ++i)
        if (j0 + i < n1)
#pragma unroll
          for (int r = 0; r < R; ++r) fma4(acc[r], v[i], b[i][r]);
    }
    __syncwarp(mask);
    stage_tile(stage, base + STAGES * T);
    stage ^= 1;
  }
  cp_async_wait<0>();

  float* crow = C + (int64_t)row * K + lane * 4;
#pragma unroll
  for (int r = 0; r < R; ++r) st_stream(crow + r * W * 4, acc[r]);
}

// ---- K = 128 with the rows of B fetched by TMA ----------------------------------------------------
// Same chunks, same order of additions and same settlement as spmm_warp_kernel at K = 128; what differs is
// how a row of B (512 bytes) reaches the warp.  Lane 0 names four rows at a time to the tensor memory
// accelerator (cp.async.bulk.tensor ... tile::gather4 on a tensor map of B whose box is one row), which
// writes them into a ring of kTmaRing 2 KB buffers private to the warp and signals an mbarrier per buffer;
// the warp reads each row back with one 16-byte shared-memory load per lane.  The gathers of up to
// kTmaRing groups are in flight while the warp multiplies, whatever its register budget, and they occupy
// neither the load/store unit's global path nor registers while they travel.
//
// The chunk's (column, value) pairs are staged whole (a chunk of nominal size S holds at most 2 S - 1
// entries, and the launcher takes plans up to S = kTmaMaxS).
// Every wait is bounded by a clock limit; a warp whose wait runs out counts that in *fallbacks, fetches
// the rest of its chunk with ordinary loads and, before it leaves, waits (bounded again) for the copies
// it still has in flight, so a fault in the protocol costs time and leaves a record but neither hangs
// nor changes the result.
#ifndef HPSPMM_TMA_RING
#define HPSPMM_TMA_RING 2
#endif
#ifndef HPSPMM_TMA_WARPS
#define HPSPMM_TMA_WARPS 8
#endif
#ifndef HPSPMM_TMA_BATCH
#define HPSPMM_TMA_BATCH 1
#endif
constexpr int kTmaBatch = HPSPMM_TMA_BATCH;        // groups issued per TMA instruction (one per lane)
constexpr int kTmaRing = HPSPMM_TMA_RING;          // 2 KB buffers per warp, a multiple of kTmaBatch
#ifndef HPSPMM_TMA_MAX_S
#define HPSPMM_TMA_MAX_S 256
#endif
constexpr int kTmaMaxS = HPSPMM_TMA_MAX_S;         // largest nominal chunk size taken
constexpr int kTmaMaxChunk = 2 * kTmaMaxS;         // a chunk holds at most 2 S - 1 entries (chunk_table_kernel)
constexpr int kTmaWarps = HPSPMM_TMA_WARPS;        // warps (= chunks) per block; three blocks per SM
constexpr int kTmaGroupBytes = 4 * 128 * 4;        // four rows of 128 floats
constexpr long long kTmaSpinLimit = 1000000000ll;  // clock cycles, about half a second
static_assert(kTmaRing % kTmaBatch == 0 && kTmaRing >= 2 * kTmaBatch, "ring = whole batches, at least two");
constexpr int kTmaSmemPerWarp = kTmaRing * kTmaGroupBytes + kTmaMaxChunk * 8 + kTmaRing * 8;

__device__ __forceinline__ uint32_t smem_addr_of(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// the slow side of a wait: polls until the phase completes or the clock limit passes
__device__ __noinline__ bool mbar_wait_slow(uint32_t bar, uint32_t parity) {
  const long long t0 = clock64();
  for (unsigned n = 1;; ++n) {
    if (mbar_try(bar, parity)) return true;
    if ((n & 63u) == 0 && clock64() - t0 > kTmaSpinLimit) return false;
  }
}

__device__ __forceinline__ bool mbar_wait_limited(uint32_t bar, uint32_t parity) {
  if (mbar_try(bar, parity)) return true;   // the copy has usually landed: no clock read, no loop
  return mbar_wait_slow(bar, parity);
}

__global__ void __launch_bounds__(kTmaWarps * 32, 3)
spmm_tma_kernel(const __grid_constant__ CUtensorMap map_b, int M, int n_chunks, int n_chunk_blocks,
                const int* __restrict__ row_ptr, const int* __restrict__ col_idx,
                const float* __restrict__ vals, const float* __restrict__ B, float* __restrict__ C,
                const int* __restrict__ chunk_start, const int* __restrict__ chunk_row,
                float* __restrict__ carry_val, const int* __restrict__ chunk_order, int S,
                int* __restrict__ run_counter, const int* __restrict__ nz_id, const int* __restrict__ nz_end,
                const int* __restrict__ chunk_ri, int* __restrict__ fallbacks) {
  constexpr int KW = 128;
  constexpr int64_t K = KW;
  extern __shared__ __align__(1024) unsigned char tma_smem[];
  if ((int)blockIdx.x >= n_chunk_blocks) {
    zero_empty_rows<KW>(M, KW, row_ptr, C, blockIdx.x - n_chunk_blocks, gridDim.x - n_chunk_blocks, kTmaWarps * 32);
    return;
  }
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int slot = blockIdx.x * kTmaWarps + warp;
  if (slot >= n_chunks) return;
  const int chunk = chunk_order != nullptr ? __ldg(chunk_order + slot) : slot;

  // this warp's part of shared memory: ring buffers (1 KB aligned), staged entries, barriers
  unsigned char* ring = tma_smem + (size_t)warp * (kTmaRing * kTmaGroupBytes);
  int2* ent = reinterpret_cast<int2*>(tma_smem + (size_t)kTmaWarps * (kTmaRing * kTmaGroupBytes)) + warp * kTmaMaxChunk;
  uint64_t* full = reinterpret_cast<uint64_t*>(tma_smem + (size_t)kTmaWarps * (kTmaRing * kTmaGroupBytes + kTmaMaxChunk * 8)) +
                   warp * kTmaRing;

  const int n0 = __ldg(chunk_start + chunk);
  const int n1 = __ldg(chunk_start + chunk + 1);
  const int len = n1 - n0;                  // < kTmaMaxChunk: the launcher checks the plan's chunk size
  const int n_groups = (len + 3) >> 2;
  int ri = __ldg(chunk_ri + chunk);
  int row = __ldg(nz_id + ri);
  int row_end = __ldg(nz_end + ri);

  for (int i = lane; i < n_groups * 4; i += 32) {
    if (i < len) {
      cp_async_4(&ent[i].x, col_idx + n0 + i);
      cp_async_4(&ent[i].y, vals + n0 + i);
    } else {
      ent[i] = make_int2(0, 0);             // past the chunk: row 0 is fetched and not used
    }
  }
  cp_async_commit();
  if (lane == 0) {
#pragma unroll
    for (int b = 0; b < kTmaRing; ++b)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr_of(&full[b])), "r"(1) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  cp_async_wait<0>();
  __syncwarp();

  // lane 0: fetch the four rows of group g into buffer g % kTmaRing
  auto issue = [&](int g) {
    const int b = g % kTmaRing;
    const uint32_t bar = smem_addr_of(&full[b]);
    const int4 c01 = *reinterpret_cast<const int4*>(&ent[4 * g]);
    const int4 c23 = *reinterpret_cast<const int4*>(&ent[4 * g + 2]);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(kTmaGroupBytes) : "memory");
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cta.global.tile::gather4.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(smem_addr_of(ring + (size_t)b * kTmaGroupBytes)),
        "l"(&map_b), "r"(0), "r"(c01.x), "r"(c01.z), "r"(c23.x), "r"(c23.z), "r"(bar)
        : "memory");
  };
  // One TMA instruction costs the SM about as much as five gather4 operations, so the lanes 0 .. kTmaBatch-1
  // issue one group each with a single instruction, every kTmaBatch groups.
  const int ahead = n_groups < kTmaRing ? n_groups : kTmaRing;
  for (int g0 = 0; g0 < ahead; g0 += kTmaBatch)
    if (lane < kTmaBatch && g0 + lane < ahead) issue(g0 + lane);
  int issued = ahead;                        // groups handed to the TMA so far (warp-uniform)

  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  auto finish_row = [&]() {
    st_stream(C + (int64_t)row * K + lane * 4, acc);
    acc = make_float4(0.f, 0.f, 0.f, 0.f);
    ++ri;
    row = __ldg(nz_id + ri);
    row_end = __ldg(nz_end + ri);
  };

  bool by_tma = true;
  int pending_from = 0;                      // first group whose copy was never seen to land
  const uint32_t bar0 = smem_addr_of(full);
  // one group: wait for its buffer, read the four rows, hand the buffer back to the TMA, multiply
  auto do_group = [&](int g, int b, uint32_t parity) {
    float4 rows4[4];
    float v[4];
    const int4 e01 = *reinterpret_cast<const int4*>(&ent[4 * g]);       // (col, val) x 2, broadcast
    const int4 e23 = *reinterpret_cast<const int4*>(&ent[4 * g + 2]);
    v[0] = __int_as_float(e01.y), v[1] = __int_as_float(e01.w);
    v[2] = __int_as_float(e23.y), v[3] = __int_as_float(e23.w);
    if (by_tma) {
      const bool ok = mbar_wait_limited(bar0 + 8u * (uint32_t)b, parity);
      by_tma = __all_sync(0xffffffffu, ok);
      if (!by_tma) {
        pending_from = g;
        if (lane == 0) atomicAdd(fallbacks, 1);
      }
    }
    if (by_tma) {
      const float4* src = reinterpret_cast<const float4*>(ring + (size_t)b * kTmaGroupBytes) + lane;
#pragma unroll
      for (int i = 0; i < 4; ++i) rows4[i] = src[i * 32];
      __syncwarp();                          // every lane has read the buffer before it is refilled
      if ((b + 1) % kTmaBatch == 0 && issued < n_groups) {
        // the kTmaBatch buffers of groups g - kTmaBatch + 1 .. g are free: refill them with the next groups
        // (the warp's reads of these buffers are ordered before this point by the __syncwarp above; the
        // refill is ordered after it by program order, as in any mbarrier-released TMA ring)
        const int n_new = min(kTmaBatch, n_groups - issued);
        if (lane < n_new) issue(issued + lane);
        issued += n_new;
      }
    } else {
      const int cols[4] = {e01.x, e01.z, e23.x, e23.z};
#pragma unroll
      for (int i = 0; i < 4; ++i) rows4[i] = ld_gather_plain(B + (int64_t)cols[i] * K + lane * 4);
    }
    const int j0 = n0 + 4 * g;
    if (j0 + 4 <= n1 && row_end >= j0 + 4) {
#pragma unroll
      for (int i = 0; i < 4; ++i) fma4(acc, v[i], rows4[i]);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int j = j0 + i;
        if (j < n1) {
          while (row_end <= j) finish_row();   // warp-uniform
          fma4(acc, v[i], rows4[i]);
        }
      }
    }
  };
  // the ring is walked in whole turns so that a group's buffer index is a compile-time constant
  for (int turn = 0; turn * kTmaRing < n_groups; ++turn) {
    const uint32_t parity = (uint32_t)turn & 1u;
#pragma unroll
    for (int b = 0; b < kTmaRing; ++b) {
      const int g = turn * kTmaRing + b;
      if (g < n_groups) do_group(g, b, parity);
    }
  }
  if (!by_tma) {
    // copies still in flight target this block's shared memory: let them land before the warp leaves
    for (int g = pending_from; g < issued; ++g)
      mbar_wait_limited(smem_addr_of(&full[g % kTmaRing]), (uint32_t)(g / kTmaRing) & 1u);
  }

  const bool hands_on = row_end != n1;   // the chunk ends inside `row`
  if (!hands_on)
    st_stream(C + (int64_t)row * K + lane * 4, acc);
  else
    *reinterpret_cast<float4*>(carry_val + (int64_t)chunk * K + lane * 4) = acc;
  const int r0 = __ldg(chunk_row + chunk);
  const int r0_start = __ldg(row_ptr + r0), r0_end = __ldg(row_ptr + r0 + 1);
  const bool stores_split_row = r0_start < n0 && r0_end <= n1;   // began in an earlier chunk, ends here
  if (!hands_on && !stores_split_row) return;
  settle_split_rows<4, 32, 1>(stores_split_row, r0, r0_start, r0_end, hands_on, row, __ldg(row_ptr + row), row_end, chunk,
                              S, carry_val, C, run_counter, KW, KW);
}

// ---- row-split kernel for any other K: one warp per row ------------------------------------------
// Lane l owns columns kb + (s*32 + l)*VEC .. +VEC-1 for s < NS, where kb = blockIdx.y * (32*VEC*NS).
// VEC = 4 needs K % 4 == 0.
template <int VEC, int NS>
__global__ void __launch_bounds__(kBlockThreads)
spmm_rowsplit_any_kernel(int M, int K, const int* __restrict__ row_ptr, const int* __restrict__ col_idx,
                         const float* __restrict__ vals, const float* __restrict__ B, float* __restrict__ C) {
  const int lane = threadIdx.x & 31;
  const int row = (int)(((int64_t)blockIdx.x * kBlockThreads + threadIdx.x) >> 5);
  if (row >= M) return;
  const int kb = blockIdx.y * (32 * VEC * NS);
  const int n0 = __ldg(row_ptr + row);
  const int n1 = __ldg(row_ptr + row + 1);

  float acc[NS][VEC];
  int colbase[NS];
  bool live[NS];
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    colbase[s] = kb + (s * 32 + lane) * VEC;
    live[s] = colbase[s] < K;  // VEC == 4 implies K % 4 == 0, so the whole vector is inside
#pragma unroll
    for (int x = 0; x < VEC; ++x) acc[s][x] = 0.f;
  }
  for (int base = n0; base < n1; base += 32) {
    const int jj = base + lane;
    int mycol = 0;
    float myval = 0.f;
    if (jj < n1) {
      mycol = ld_stream(col_idx + jj);
      myval = ld_stream(vals + jj);
    }
    const int cnt = min(32, n1 - base);
    for (int i = 0; i < cnt; ++i) {
      const int c = __shfl_sync(0xffffffffu, mycol, i);
      const float v = __shfl_sync(0xffffffffu, myval, i);
      const float* brow = B + (int64_t)c * K;
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        if (!live[s]) continue;
        if (VEC == 4) {
          const float4 t = __ldg(reinterpret_cast<const float4*>(brow + colbase[s]));
          acc[s][0] = fmaf(v, t.x, acc[s][0]);
          acc[s][VEC > 1 ? 1 : 0] = fmaf(v, t.y, acc[s][VEC > 1 ? 1 : 0]);
          acc[s][VEC > 2 ? 2 : 0] = fmaf(v, t.z, acc[s][VEC > 2 ? 2 : 0]);
          acc[s][VEC > 3 ? 3 : 0] = fmaf(v, t.w, acc[s][VEC > 3 ? 3 : 0]);
        } else {
#pragma unroll
          for (int x = 0; x < VEC; ++x) acc[s][x] = fmaf(v, __ldg(brow + colbase[s] + x), acc[s][x]);
        }
      }
    }
  }
  float* dst = C + (int64_t)row * K;
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    if (!live[s]) continue;
#pragma unroll
    for (int x = 0; x < VEC; ++x) dst[colbase[s] + x] = acc[s][x];
  }
}

template <int W>
void launch_rowsplit(bool hint, int M, const int32_t* row_ptr, const int32_t* col_idx, const float* vals,
                     const float* B, float* C, cudaStream_t stream) {
  constexpr int workers_per_block = kBlockThreads / W;
  const unsigned grid = (unsigned)(((int64_t)M + workers_per_block - 1) / workers_per_block);
  if (hint)
    spmm_rowsplit_kernel<W, 1, 8, 4, true><<<grid, kBlockThreads, 0, stream>>>(M, row_ptr, col_idx, vals, B, C);
  else
    spmm_rowsplit_kernel<W, 1, 8, 4, false><<<grid, kBlockThreads, 0, stream>>>(M, row_ptr, col_idx, vals, B, C);
}

int run_rowsplit(hpspmm_ctx* ctx, bool hint, int M, int64_t K, const int32_t* row_ptr, const int32_t* col_idx,
                 const float* vals, const float* B, float* C, cudaStream_t stream) {
  if (K == 32) {
    launch_rowsplit<8>(hint, M, row_ptr, col_idx, vals, B, C, stream);
  } else if (K == 64) {
    launch_rowsplit<16>(hint, M, row_ptr, col_idx, vals, B, C, stream);
  } else if (K == 128) {
    launch_rowsplit<32>(hint, M, row_ptr, col_idx, vals, B, C, stream);
  } else {
    const int kblock = 32 * 4 * ((K & 3) == 0 ? 4 : 1);
    const int64_t n_kblocks = (K + kblock - 1) / kblock;
    if (n_kblocks > 65535) return HPSPMM_ERR_UNSUPPORTED;
    const dim3 grid((unsigned)((M + kBlockThreads / 32 - 1) / (kBlockThreads / 32)), (unsigned)n_kblocks, 1);
    if ((K & 3) == 0)
      spmm_rowsplit_any_kernel<4, 4><<<grid, kBlockThreads, 0, stream>>>(M, (int)K, row_ptr, col_idx, vals, B, C);
    else
      spmm_rowsplit_any_kernel<1, 4><<<grid, kBlockThreads, 0, stream>>>(M, (int)K, row_ptr, col_idx, vals, B, C);
  }
  ctx->launches++;
  HPSPMM_CUDA_TRY(ctx, cudaGetLastError());
  return HPSPMM_OK;
}

inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

typedef CUresult (*tensor_map_encode_fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                         const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                         CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

tensor_map_encode_fn tensor_map_encoder() {
  static std::once_flag once;
  static tensor_map_encode_fn fn = nullptr;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &found) == cudaSuccess &&
        found == cudaDriverEntryPointSuccess)
      fn = (tensor_map_encode_fn)p;
  });
  return fn;
}

// The K = 128 product with B fetched by TMA.  Returns 1 when this path cannot take the call (no encoder in
// the driver, a chunk size beyond what the kernel stages, a B the tensor map refuses): the caller then runs
// the ordinary kernel.  0 = launched, negative = error.
int launch_spmm_tma(hpspmm_ctx* ctx, int m, int nc, int64_t rows_b, const int32_t* row_ptr, const int32_t* col_idx,
                    const float* vals, const float* B, float* C, const int32_t* chunk_start,
                    const int32_t* chunk_row, float* carry_val, const int32_t* chunk_order, int S,
                    int* run_counter, const hpspmm_plan* rows, cudaStream_t stream) {
  if (S <= 0 || S > kTmaMaxS || rows_b <= 0) return 1;
  tensor_map_encode_fn enc = tensor_map_encoder();
  if (!enc) return 1;
  CUtensorMap map_b;
  const cuuint64_t gdim[2] = {128, (cuuint64_t)rows_b};
  const cuuint64_t gstride[1] = {512};
  const cuuint32_t box[2] = {128, 1};   // gather4: one row per box, four boxes per operation
  const cuuint32_t estride[2] = {1, 1};
  if (enc(&map_b, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(B), gdim, gstride, box, estride,
          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return 1;
  constexpr int smem = kTmaWarps * kTmaSmemPerWarp;
  // per call: the attribute belongs to the current device's context, and a process may drive several GPUs
  if (cudaFuncSetAttribute(spmm_tma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) {
    cudaGetLastError();
    return 1;
  }
  const int n_chunk_blocks = (nc + kTmaWarps - 1) / kTmaWarps;
  int n_zero_blocks = (m + kTmaWarps * 32 - 1) / (kTmaWarps * 32);
  const int cap = ctx->sm_count * 4;
  if (n_zero_blocks > cap) n_zero_blocks = cap;
  const unsigned grid = (unsigned)(n_chunk_blocks + n_zero_blocks);
  if (grid == 0) return 0;
  spmm_tma_kernel<<<grid, kTmaWarps * 32, smem, stream>>>(map_b, m, nc, n_chunk_blocks, row_ptr, col_idx, vals, B, C,
                                                          chunk_start, chunk_row, carry_val, chunk_order, S,
                                                          run_counter, rows->nz_id, rows->nz_end, rows->chunk_ri,
                                                          ctx->flag + HPSPMM_FLAG_TMA_FALLBACKS);
  ctx->launches++;
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    hpspmm_set_err(ctx, HPSPMM_ERR_CUDA, "spmm_tma_kernel launch", e);
    return -1;
  }
  return 0;
}

}  // namespace

// Nominal chunk size of the kernels that probe row_ptr or reduce into C (the allocation-free entry, the COO
// product): measured best on B200 (R-MAT scale 20) at 128 / 160 / 256 entries for K = 32 / 64 / 128.
static int32_t probing_chunk_nnz(int64_t K) {
  if (K <= 32) return 128;
  if (K <= 64) return 160;
  return 256;
}

int32_t hpspmm_default_chunk_nnz(int64_t K, int64_t nnz) {
  // Larger chunks amortise the per-chunk prologue and split fewer rows; but the SDDMM shares the plan, and there a chunk
  // of very short rows waits once per row, so its time turns up with the longest such chunk once chunks are few.
  // Power-law graphs, S = 128 / 192 / 256 / 320 / 384 / 512 in us, product and SDDMM:
  //   4 M entries,  K = 64: 83 / 80 / 75 / 79 / 80 / 82        and 75 / 74 / 88 / 103 / 101 / 98
  //   5 M entries,  K = 32: 66 / 61 / 61 / 57 / 58 / 64        and 57 / 56 / 63 / 77 / 90 / 72
  //   8 M entries,  K = 32: 110 / 97 / 93 / 93 / 90 / 87       and 94 / 92 / 91 / 92 / 103 / 134
  //   12 M entries, K = 32: 164 / 144 / 135 / 133 / 133 / 132  and 145 / 138 / 136 / 135 / 135 / 137
  //   16 M entries, K = 64: 333 / 322 / 305 / 297 / 293 / 297  and 294 / 293 / 292 / 294 / 299 / 303
  //   16 M entries, K = 128: 566 / 567 / 546 / - / 550 / 526   and 523 / 563 / 572 / 566 / 537 / 561
  // A caller that builds a plan for products only can ask for more (hpspmm_opts.chunk_nnz).
  // Below 2.4 M entries there are at most a few waves of chunks (5,300 warps of the fixed widths are resident), and the
  // time is that of the longest chunk: a chain of gather round trips.  Measured in us at S = 32 / 64 / 128 / 256, rows of 16 entries on average,
  // uniform and power-law columns: 12 K entries, K = 32: 3.7 / 4.5 / 6.3 / 10.1 and 6.6 / 7.7 / 10.3 / 13.9;
  // 300 K, K = 64: 10.2 / 8.3 / 10.3 / 16.3 and 14.2 / 12.9 / 15.6 / 24.2; 1 M, K = 64: 24.3 / 21.0 / 21.4 / 22.7 and
  // 37.5 / 26.7 / 23.8 / 32.2 (smaller chunks split more rows, and every split costs an exchange through memory).
  // Beyond 64 columns a split costs as much but saves less, so chunks of 128 begin earlier.
  if (nnz < 32000) return 32;
  if (nnz < (K > 64 ? 150000 : 500000)) return 64;
  if (nnz < 2400000) return 128;
  const int32_t floor_s = probing_chunk_nnz(K);
  const int32_t best = K <= 32 ? 384 : (K <= 64 ? 320 : 256);
  const int64_t want = nnz / 24000 / 32 * 32;
  int64_t s = want < floor_s ? floor_s : want;
  if (s > best) s = best;
  return (int32_t)s;
}

int32_t hpspmm_coo_chunk_nnz(int64_t K, int64_t nnz) {
  // 4 M triples of a power-law graph, S = 64 / 128 / 160 / 256: K = 32 56.0 / 56.2 / 57.6 / 63.0 us, K = 64 78.6 / 77.3 /
  // 78.1 / 83.2; below 768 K triples as many chunks as the GPU has warps, down to 32 triples.
  const int32_t best = K <= 128 ? 128 : 256;
  const int64_t want = nnz / 6000 / 32 * 32;
  return (int32_t)(want < 32 ? 32 : (want > best ? best : want));
}

int hpspmm_vector_width(int64_t K, uintptr_t addresses) {
  // K % 4 == 0 is refused by the entry points unless the operands are 16-byte aligned
  return (K & 3) == 0 ? 4 : ((K & 1) == 0 && (addresses & 7) == 0 ? 2 : 1);
}

hpspmm_spmm_shape hpspmm_choose_shape(int VEC, int64_t cols, int widest, bool hint) {
  hpspmm_spmm_shape sh;
  sh.VEC = VEC;
  sh.hint = hint;
  sh.lat = false;
  sh.mid = false;
  if (cols > widest) cols = widest;
  const int vecs = (int)((cols + VEC - 1) / VEC);
  sh.W = VEC == 1 ? (vecs <= 1 ? 1 : 4) : 2;
  while (sh.W < 32 && sh.W < vecs) sh.W *= 2;
  sh.R = (vecs + 31) / 32;
  // 33 to 48 narrow vectors: two groups of 16 lanes with three vectors each leave no lane idle and read two entries per
  // step (4 M entries, uniform columns: K = 47 107 -> 89 us, K = 66 148 -> 132 us; a power-law graph gains nothing)
  if (vecs > 32 && vecs <= 48) sh.W = 16, sh.R = 3;
  // 17 to 24 wide vectors: four groups of 8 lanes, for the same reason.  R-MAT scale 20 / 8 M uniform entries: K = 96
  // 484 -> 440 / 200 -> 175 us; and with 16 lanes K = 160 812 -> 707 / 467 -> 378 us, K = 192 875 -> 796 / 548 -> 482 us.
  // (25 to 32 vectors lose: K = 100 516 -> 529 us, K = 128 524 -> 544 us, the rows' ends then cost exchanges.)
  if (VEC == 4 && vecs > 16 && vecs <= 24) sh.W = 8, sh.R = 3;
  return sh;
}

namespace {

int check_spmm_args(hpspmm_ctx* ctx, int64_t M, int64_t N, int64_t K, int64_t nnz,
                    const void* row_ptr, const void* col_idx, const void* vals, const void* B,
                    const void* C) {
  HPSPMM_REQUIRE(ctx, ctx != nullptr, "null context");
  HPSPMM_REQUIRE(ctx, M >= 0 && N >= 0 && nnz >= 0, "negative size");
  HPSPMM_REQUIRE(ctx, K >= 1, "K must be >= 1");
  // entry positions are 32-bit and the kernels look up to one tile past a chunk's end
  if (M > 2147483646ll || N > 2147483647ll || nnz > 2147483647ll - 4096 || K > (1 << 20)) {
    snprintf(ctx->err, sizeof(ctx->err), "sizes beyond 32-bit CSR indices");
    return HPSPMM_ERR_UNSUPPORTED;
  }
  HPSPMM_REQUIRE(ctx, row_ptr != nullptr, "null row_ptr");
  HPSPMM_REQUIRE(ctx, nnz == 0 || (col_idx && vals && B), "null operand");
  HPSPMM_REQUIRE(ctx, M == 0 || C != nullptr, "null output");
  if ((K & 3) == 0 && (((uintptr_t)B & 15u) || ((uintptr_t)C & 15u))) {
    snprintf(ctx->err, sizeof(ctx->err), "dense operands must be 16-byte aligned");
    return HPSPMM_ERR_INVALID;
  }
  return HPSPMM_OK;
}

// Widest slab of a product's columns.  With wide vectors one pass over up to 512 columns holds two to four vectors of a
// row per lane, so only one or two entries are in flight, and all of B competes for the L2 cache.  Passes of 128 columns
// read the small sparse operand again instead, keep four entries in flight and need a part of B at a time.
// One pass -> passes in us:
//   uniform rows:     1 M entries, 62.5 K rows, K = 448 202 -> 129;  2 M, 200 K rows, K = 256 236 -> 195, 320 347 -> 258,
//                     448 554 -> 364;  4 M, 250 K rows, K = 256 483 -> 417, 320 685 -> 488, 512 1189 -> 798
//   power-law graphs: 1.2 M, 60 K rows, K = 392 136 -> 141, 512 148 -> 142;  4 M, 250 K rows, K = 392 479 -> 446, 512 548 ->
//                     501, and without a plan 590 -> 557; below 384 columns about level with a plan, and without one, where the
//                     chunks are not ordered by cost and every pass ends on its own last ones, behind (4 M, K = 300 +6 %)
// 300 K entries, K = 512: 37 -> 47, so with few chunks one pass stays.
int widest_slab(int sm_count, int VEC, int64_t K, int64_t n_chunks, bool even) {
  if (VEC == 4 && ((K > 384 && n_chunks > sm_count * 48ll) || (K >= 256 && even && n_chunks > sm_count * 64ll))) return 128;
  return hpspmm_widest_slab(VEC);
}

// The launch of a product that begins at column `off`: how many columns it takes (*cols) and its shape.
hpspmm_spmm_shape shape_of_launch(int sm_count, int VEC, int K, int off, int64_t n_chunks, bool even, bool hint, int* cols) {
  const int widest = widest_slab(sm_count, VEC, K, n_chunks, even);
  *cols = hpspmm_launch_cols(K, off, widest);
  hpspmm_spmm_shape sh = hpspmm_choose_shape(VEC, *cols, widest, hint);
  // Few chunks: registers are plenty, so a warp keeps 8 to 32 gather steps in flight instead of 4 (the additions keep
  // their order).  67.6 K entries in chunks of 64: 6.1 -> 5.6 us at K = 64, 9.1 -> 7.2 us at K = 128; with more chunks
  // than these builds have resident warps they lose (300 K entries, K = 64: 8.3 -> 10.5 us).
  sh.lat = n_chunks <= sm_count * (sh.W <= 8 ? 24 : 16);
  // A warp over 97 to 128 or 193 to 256 columns has four or two entries in flight.  With twice as many 24 warps fit on an SM
  // instead of 36, which pays where the chunks are about one or two waves of those.  Chunks per SM: 17.7 to 22 / 37 to 42,
  // power-law and uniform graphs of 335 K to 800 K entries, plan, 36 -> 24 warps in us:
  //   K = 100  23.2 -> 21.3, 17.0 -> 15.5 / 28.0 -> 25.6, 42.8 -> 38.5;   K = 128  22.9 -> 21.3, 16.8 -> 15.7 / 31.0 -> 29.3, 46.9 -> 41.7
  //   K = 224  34.3 -> 28.2, 29.0 -> 23.6 / 57.0 -> 48.3, 49.5 -> 42.7;   K = 256  34.4 -> 28.6, 29.6 -> 25.8 / 59.8 -> 51.2, 53.9 -> 47.0
  // Between (30 per SM) uniform rows lose (K = 128 19.9 -> 25.4), from 53 on it is level or behind, and at up to 64 columns
  // uniform rows lose everywhere (335 K, K = 64: 8.4 -> 10.4).
  sh.mid = !sh.lat && VEC == 4 && sh.W == 32 && sh.R <= 2 &&
           (n_chunks <= sm_count * 24ll || (n_chunks > sm_count * 36ll && n_chunks <= sm_count * 48ll));
  // (one group instead of several of three vectors: rows end without an exchange, and are added up in another order)
  if (sh.lat && sh.R == 3 && sh.W < 32) sh.R = sh.W / 8, sh.W = 32;
  return sh;
}

// shared_counters: the scratch holds one counter per chunk, so the slabs of a wide product run one after the other
// even: the rows are known to be of even length (hpspmm_even_rows)
int launch_spmm(hpspmm_ctx* ctx, hpspmm_spmm_args a, bool hint, bool even, bool shared_counters, cudaStream_t s) {
  const int VEC = hpspmm_vector_width(a.K, (uintptr_t)a.B | (uintptr_t)a.C);
  int32_t* counter = a.counter;
  a.keep_b = hint ? 1 : 0;
  for (a.off = 0; a.off < a.K; a.off += a.cols) {
    const hpspmm_spmm_shape sh = shape_of_launch(ctx->sm_count, VEC, a.K, a.off, a.n_chunks, even, hint, &a.cols);
    if (!shared_counters) a.counter = counter + (int64_t)(a.off / 32) * a.n_chunks;
    const int st = VEC == 4   ? hpspmm_spmm_launch_v4(ctx, a, sh, shared_counters, s)
                   : VEC == 2 ? hpspmm_spmm_launch_v2(ctx, a, sh, shared_counters, s)
                              : hpspmm_spmm_launch_v1(ctx, a, sh, shared_counters, s);
    if (st != HPSPMM_OK) return st;
  }
  return HPSPMM_OK;
}

bool gather_hint(int64_t K, const hpspmm_opts* opts) {
  // evict-last on the gathers of B, R-MAT bench graph, on / off, one width timed alone: K = 128 0.555 / 0.591 ms,
  // K = 64 0.307 / 0.304, K = 32 0.189 / 0.1885.  Inside a step of three products run back to back K = 64 measures
  // the other way round (0.311 on, 0.313 off), so 64 columns stay on.
  const int mode = opts ? opts->b_l2_hint : 0;
  return mode == 2 || (mode == 0 && K >= 64);
}

}  // namespace

namespace {

int32_t planless_chunk_nnz(int64_t K, int64_t nnz, const hpspmm_opts* opts) {
  const int32_t S = (opts && opts->chunk_nnz > 0) ? opts->chunk_nnz : hpspmm_default_chunk_nnz(K, nnz);
  return (S + 31) / 32 * 32;
}

// Whether a product without a plan lets every warp search row_ptr for its chunk (one launch) instead of building the
// records and the list of filled rows first (two more).  A search costs a chunk 1 to 2 us of latency and the product its
// steps along row_ptr, the builders 2 to 3 us a call; with more chunks than fit on the GPU (32 warps per SM of the searching
// builds) the searches add up, and long rows gain by the records' order (pieces last).  Rows of even length gain by records
// from there on only; a power-law graph would gain below as well, but without a plan the rows are not known, and one kind
// is not to pay for the other.  Search -> records in us, chunks of 128, square matrices of 4 / 16 / 50 entries per row:
//   chunks per SM   17                                20                                24
//     uniform K=100 20.8>22.0 / 15.9>17.7 / 14.4>16.5 23.3>24.3 / 17.6>18.8 / 15.6>17.2 27.8>28.5 / 18.1>19.8 / 16.9>18.7
//     uniform K=256 43.2>45.9 / 23.5>26.1 / 23.1>25.6 49.9>52.5 / 26.7>29.3 / 25.4>27.6 64.4>65.8 / 29.7>31.9 / 27.9>30.1
//     skewed  K=100 44.5>26.3 / 27.4>23.3 / 22.2>21.8 43.7>28.1 / 31.9>24.8 / 23.1>23.8 49.5>29.3 / 32.6>26.7 / 24.6>24.6
//     skewed  K=256 55.9>39.9 / 34.7>31.4 / 27.6>31.1 56.0>41.8 / 38.5>33.4 / 29.5>33.0 65.1>49.5 / 41.3>36.3 / 32.2>34.3
//   chunks per SM   28                                32                                33
//     uniform K=32  18.1>20.8 / 11.6>13.6 /  9.3>11.3 19.5>21.2 / 12.6>13.9 /  9.8>11.9 24.2>22.1 / 15.8>14.7 / 12.8>12.2
//     uniform K=64  21.1>25.3 / 14.2>17.1 / 12.7>14.9 22.4>26.2 / 15.2>17.8 / 13.5>16.1 31.2>27.2 / 20.6>18.1 / 17.8>15.8
//     uniform K=128 37.9>40.3 / 21.6>23.3 / 20.4>22.1 42.0>44.7 / 23.8>24.9 / 21.8>23.5 62.0>46.3 / 31.6>24.5 / 28.3>23.6
//     skewed  K=64  47.9>28.9 / 29.0>23.1 / 21.9>21.3 49.2>28.8 / 30.5>23.5 / 22.9>23.3 52.3>28.9 / 35.2>25.1 / 29.3>22.7
//   chunks per SM   36                                37                                40
//     uniform K=32  25.2>22.5 / 16.5>14.8 / 13.4>12.1 25.4>24.5 / 16.6>16.4 / 13.5>14.3 26.5>25.4 / 17.0>16.9 / 13.9>14.8
//     uniform K=64  34.3>27.5 / 21.5>18.5 / 18.7>16.4 35.7>36.5 / 22.1>22.3 / 18.9>20.0 38.5>38.7 / 22.0>23.1 / 19.4>21.0
//     uniform K=128 65.9>49.1 / 33.1>26.1 / 29.8>25.2 59.2>58.6 / 32.0>31.3 / 28.1>28.5 62.2>61.4 / 32.6>32.0 / 29.3>29.3
//     skewed  K=64  55.9>30.9 / 36.7>24.2 / 30.2>24.0 62.2>32.4 / 37.5>26.9 / 29.8>24.4 55.6>31.6 / 38.0>25.2 / 30.6>25.3
//   below 32 columns rows of even length gain nothing by records before 41 per SM:
//   chunks per SM   33                                36                                40
//     uniform K=1   15.3>16.9 /  9.0>11.1 /  7.4>11.1 16.7>18.0 / 10.4>12.2 /  7.6>11.1 18.2>19.1 / 10.8>12.7 /  8.2>11.1
//     uniform K=8   21.4>21.4 / 12.2>12.9 / 10.3>11.7 22.3>22.3 / 12.9>13.5 / 10.5>12.1 23.3>23.1 / 13.2>13.6 / 11.2>12.5
//     uniform K=24  24.2>23.7 / 15.8>16.0 / 13.1>14.4 25.1>24.9 / 16.5>16.5 / 13.5>14.6 26.4>25.8 / 17.1>17.1 / 14.1>15.2
//     skewed  K=8   48.6>25.1 / 30.4>21.3 / 23.4>18.3 51.7>27.3 / 32.1>21.6 / 23.7>19.6 51.1>28.7 / 33.6>21.4 / 24.7>18.8
// (between 37 and 40 the records' product is in its second wave, and uniform rows of 16 and more entries are up to 8 % behind
// at K = 32 to 64; everything else is ahead there.)  Chunks of 64: 335 K entries (35 per SM), power-law K = 64 20.6 -> 22.1; 300 K
// (32 per SM), uniform 10.0 -> 13.4.  With very many empty rows between the entries the list pays for itself.
bool searches_for_chunks(const hpspmm_ctx* ctx, int64_t M, int64_t K, int64_t nnz, int64_t n_chunks, int32_t S) {
  return n_chunks <= ctx->sm_count * (S < 128 || K < 32 ? 40ll : 32ll) && M <= 8 * nnz;
}

// Up to here a search costs little enough to do without the records where there is no room for them: a call that is
// captured cannot allocate, and another may find the device full.
bool may_search_for_chunks(const hpspmm_ctx* ctx, int64_t M, int64_t nnz, int64_t n_chunks) {
  return n_chunks <= ctx->sm_count * 40ll && M <= 8 * nnz;
}

// Counters that are set aside at the first product of a width: enough for any later one of up to that width, so that a
// smaller call never allocates.  Beyond 512 columns as many as the call needs.
int64_t counters_to_keep(const hpspmm_ctx* ctx, int64_t K, int64_t n_counter, bool search) {
  const int64_t most = (ctx->sm_count * 40ll + 1) * hpspmm_counter_slabs(K < 512 ? K : 512);
  return search && n_counter > most ? n_counter : most;
}

// where a plan-less product keeps what it builds, inside the context's scratch
struct planless_layout {
  int64_t n_counter;
  size_t counter, carry, tiles, rec, nz, bytes;
  planless_layout(int64_t M, int64_t K, int64_t n_chunks, bool search) {
    bytes = 0;
    auto take = [&](size_t b) { const size_t at = bytes; bytes += align_up(b, 256); return at; };
    n_counter = (n_chunks + 1) * hpspmm_counter_slabs(K);
    counter = take((size_t)n_counter * 4);
    carry = take((size_t)(n_chunks + 1) * (size_t)K * 4);
    tiles = search ? 0 : take((size_t)hpspmm_row_tile_ints(M) * 4);
    rec = search ? 0 : take((size_t)(n_chunks + 1) * 32);
    nz = search ? 0 : take(hpspmm_nz_bytes(M));
  }
};

}  // namespace

extern "C" {

int hpspmm_plan_create(hpspmm_ctx* ctx, int64_t M, int64_t N, int64_t nnz, const int32_t* row_ptr,
                       const int32_t* col_idx, int64_t max_K, const hpspmm_opts* opts,
                       hpspmm_stream stream, hpspmm_plan** out) {
  HPSPMM_TRACE("hpspmm_plan_create");
  HPSPMM_REQUIRE(ctx, ctx != nullptr && out != nullptr, "null context or output");
  *out = nullptr;
  HPSPMM_REQUIRE(ctx, M >= 0 && N >= 0 && nnz >= 0 && max_K >= 1, "bad size");
  HPSPMM_REQUIRE(ctx, row_ptr != nullptr, "null row_ptr");
  if (M > 2147483646ll || nnz > 2147483647ll - 4096) return HPSPMM_ERR_UNSUPPORTED;
  int32_t S = (opts && opts->chunk_nnz > 0) ? opts->chunk_nnz : hpspmm_default_chunk_nnz(max_K, nnz);
  S = (S + 31) / 32 * 32;
  hpspmm_device_guard guard(ctx->device);
  hpspmm_plan* p = new (std::nothrow) hpspmm_plan();
  if (!p) return HPSPMM_ERR_OOM;
  memset(p, 0, sizeof(*p));
  p->device = ctx->device;
  p->sm_count = ctx->sm_count;
  p->M = M;
  p->nnz = nnz;
  p->chunk_nnz = S;
  p->max_K = max_K;
  p->n_chunks = (nnz + S - 1) / S;
  const int64_t n_counter = (p->n_chunks + 1) * hpspmm_counter_slabs(max_K);
  const size_t b_int = align_up((size_t)(p->n_chunks + 1) * 4, 256);
  const size_t b_cval = align_up((size_t)(p->n_chunks + 1) * (size_t)max_K * 4, 256);
  const size_t b_count = align_up((size_t)n_counter * 4, 256);
  const size_t b_row = align_up((size_t)(M + 2) * 4, 256);         // one slot per row + sentinel
  const size_t b_nz = align_up(hpspmm_nz_bytes(M), 256);
  const size_t b_rec = align_up((size_t)(p->n_chunks + 1) * 32, 256);
  // the builders' own scratch lives in the context and is free again afterwards
  const size_t b_sort = hpspmm_order_scratch_bytes(p->n_chunks);
  const size_t b_tiles = align_up((size_t)hpspmm_row_tile_ints(M) * 4, 256);
  p->bytes = 4 * b_int + b_cval + b_count + 2 * b_row + b_nz + b_rec;
  char* base = nullptr;
  cudaError_t e = hpspmm_device_malloc((void**)&base, p->bytes);
  if (e != cudaSuccess) {
    delete p;
    return hpspmm_set_err(ctx, HPSPMM_ERR_OOM, "plan cudaMalloc", e);
  }
  char* at = base;
  auto take = [&](size_t bytes) { char* r = at; at += bytes; return r; };
  p->chunk_start = (int32_t*)take(b_int);
  p->chunk_row = (int32_t*)take(b_int);
  p->chunk_order = (int32_t*)take(b_int);
  p->chunk_ri = (int32_t*)take(b_int);
  p->carry_val = (float*)take(b_cval);
  p->run_counter = (int32_t*)take(b_count);
  p->nz_id = (int32_t*)take(b_row);
  p->nz_end = (int32_t*)take(b_row);
  p->nz = (int2*)take(b_nz);
  p->rec = (int4*)take(b_rec);
  cudaStream_t s = (cudaStream_t)stream;
  int split = 0;
  int st = hpspmm_ensure_scratch(ctx, b_sort + b_tiles + b_rec);
  char* scratch = (char*)ctx->scratch;
  int4* rec_by_chunk = (int4*)(scratch + b_sort + b_tiles);
  if (st == HPSPMM_OK) e = cudaMemsetAsync(ctx->flag, 0, sizeof(int), s);
  if (st == HPSPMM_OK && e == cudaSuccess) e = cudaMemsetAsync(p->chunk_start, 0, 4, s);
  if (st == HPSPMM_OK && e == cudaSuccess) e = cudaMemsetAsync(p->run_counter, 0, b_count, s);
  if (st == HPSPMM_OK && e == cudaSuccess)
    st = hpspmm_build_structure(ctx, M, nnz, row_ptr, S, p->n_chunks, p->nz, rec_by_chunk, (int32_t*)(scratch + b_sort),
                                hpspmm_structure_tables{p->chunk_start, p->chunk_row, p->chunk_ri, p->nz_id, p->nz_end,
                                                        ctx->flag}, s);
  if (st == HPSPMM_OK && e == cudaSuccess && M > 0)
    st = hpspmm_order_chunks_by_cost(ctx, M, N, p->n_chunks, row_ptr, col_idx, p->chunk_start, p->chunk_row,
                                     p->chunk_order, scratch, s);
  if (st == HPSPMM_OK && e == cudaSuccess && M > 0)
    st = hpspmm_order_records(ctx, p->n_chunks, p->chunk_order, rec_by_chunk, p->rec, s);
  if (e == cudaSuccess && st == HPSPMM_OK)
    e = cudaMemcpyAsync(&split, ctx->flag, sizeof(int), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess && st == HPSPMM_OK) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess || st != HPSPMM_OK) {
    cudaFree(base);
    delete p;
    return e != cudaSuccess ? hpspmm_set_err(ctx, HPSPMM_ERR_CUDA, "plan build", e) : st;
  }
  p->n_split_chunks = split;
  *out = p;
  return HPSPMM_OK;
}

int hpspmm_plan_destroy(hpspmm_ctx* ctx, hpspmm_plan* plan) {
  if (!plan) return HPSPMM_OK;
  hpspmm_device_guard guard(plan->device);
  if (plan->chunk_start) cudaFree(plan->chunk_start);
  delete plan;
  (void)ctx;
  return HPSPMM_OK;
}

int hpspmm_plan_info(const hpspmm_plan* plan, int64_t* n_chunks, int64_t* n_split_chunks,
                     int64_t* chunk_nnz, int64_t* scratch_bytes) {
  if (!plan) return HPSPMM_ERR_INVALID;
  if (n_chunks) *n_chunks = plan->n_chunks;
  if (n_split_chunks) *n_split_chunks = plan->n_split_chunks;
  if (chunk_nnz) *chunk_nnz = plan->chunk_nnz;
  if (scratch_bytes) *scratch_bytes = (int64_t)plan->bytes;
  return HPSPMM_OK;
}

int hpspmm_spmm_kernel_signature(const hpspmm_plan* plan, int64_t K, int32_t b_l2_hint, char* buf, size_t len) {
  if (!buf || len == 0 || K < 1) return HPSPMM_ERR_INVALID;
  const int VEC = hpspmm_vector_width(K, 0);
  const hpspmm_opts o = {0, 0, b_l2_hint, 0};
  const bool hint = gather_hint(K, &o);
  int cols = 0;
  const bool fits = plan != nullptr && K <= plan->max_K && K <= (1 << 20);
  const hpspmm_spmm_shape sh =
      fits ? shape_of_launch(plan->sm_count, VEC, (int)K, 0, plan->n_chunks, hpspmm_even_rows(plan), hint, &cols)
           : hpspmm_choose_shape(VEC, K, hpspmm_widest_slab(VEC), hint);
  // (mid only where it is set: captures on file were taken of builds without it)
  snprintf(buf, len, "spmm_warp_kernel<%d,%d,%d> K=%lld few=%d%s hint=%d chunk_nnz=%d", sh.VEC, sh.W, sh.R, (long long)K,
           sh.lat ? 1 : 0, sh.mid ? " mid=1" : "", sh.hint ? 1 : 0,
           plan ? (int)plan->chunk_nnz : (int)hpspmm_default_chunk_nnz(K, 0));
  return HPSPMM_OK;
}

int hpspmm_plan_tables(const hpspmm_plan* plan, const int32_t** chunk_start, const int32_t** chunk_row,
                       const int32_t** chunk_order) {
  if (!plan) return HPSPMM_ERR_INVALID;
  if (chunk_start) *chunk_start = plan->chunk_start;
  if (chunk_row) *chunk_row = plan->chunk_row;
  if (chunk_order) *chunk_order = plan->chunk_order;
  return HPSPMM_OK;
}

int hpspmm_plan_row_list(const hpspmm_plan* plan, const int32_t** nz_id, const int32_t** nz_end,
                         const int32_t** chunk_ri) {
  if (!plan) return HPSPMM_ERR_INVALID;
  if (nz_id) *nz_id = plan->nz_id;
  if (nz_end) *nz_end = plan->nz_end;
  if (chunk_ri) *chunk_ri = plan->chunk_ri;
  return HPSPMM_OK;
}

int hpspmm_spmm_csr_f32(hpspmm_ctx* ctx, const hpspmm_plan* plan, int64_t M, int64_t N, int64_t K,
                        int64_t nnz, const int32_t* row_ptr, const int32_t* col_idx,
                        const float* vals, const float* B, float* C, const hpspmm_opts* opts,
                        hpspmm_stream stream) {
  HPSPMM_TRACE("hpspmm_spmm_csr_f32");
  int st = check_spmm_args(ctx, M, N, K, nnz, row_ptr, col_idx, vals, B, C);
  if (st != HPSPMM_OK) return st;
  if (M == 0) return HPSPMM_OK;
  hpspmm_device_guard guard(ctx->device);
  cudaStream_t s = (cudaStream_t)stream;
  const bool hint = gather_hint(K, opts);
  const int algo = opts ? opts->algo : HPSPMM_ALGO_AUTO;
  if (algo == HPSPMM_ALGO_ROW_SPLIT) return run_rowsplit(ctx, hint, (int)M, K, row_ptr, col_idx, vals, B, C, s);
  HPSPMM_REQUIRE(ctx, algo == HPSPMM_ALGO_AUTO || algo == HPSPMM_ALGO_BALANCED || algo == HPSPMM_ALGO_TMA,
                 "unknown algo");
  hpspmm_spmm_args a;
  memset(&a, 0, sizeof(a));
  a.M = (int)M, a.K = (int)K;
  a.row_ptr = row_ptr, a.col_idx = col_idx, a.vals = vals, a.B = B, a.C = C;
  if (plan) {
    HPSPMM_REQUIRE(ctx, plan->M == M && plan->nnz == nnz, "plan built for another matrix");
    HPSPMM_REQUIRE(ctx, K <= plan->max_K, "K exceeds the plan's max_K");
    HPSPMM_REQUIRE(ctx, plan->device == ctx->device, "plan built on another device");
    if (algo == HPSPMM_ALGO_TMA && K == 128) {
      // B through the tensor memory accelerator; falls through when that path declines
      const int r = launch_spmm_tma(ctx, (int)M, (int)plan->n_chunks, N, row_ptr, col_idx, vals, B, C,
                                    plan->chunk_start, plan->chunk_row, plan->carry_val, plan->chunk_order,
                                    plan->chunk_nnz, plan->run_counter, plan, s);
      if (r == 0) return HPSPMM_OK;
      if (r < 0) return HPSPMM_ERR_CUDA;   // the launcher has recorded the message
    }
    a.n_chunks = (int)plan->n_chunks, a.S = plan->chunk_nnz;
    a.rec = plan->rec, a.nz = plan->nz, a.carry = plan->carry_val, a.counter = plan->run_counter;
    return launch_spmm(ctx, a, hint, hpspmm_even_rows(plan), false, s);
  }
  const int32_t S = planless_chunk_nnz(K, nnz, opts);
  const int64_t n_chunks = (nnz + S - 1) / S;
  bool search = searches_for_chunks(ctx, M, K, nnz, n_chunks, S);
  planless_layout lay(M, K, n_chunks, search);
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &capture) != cudaSuccess) cudaGetLastError();
  const bool eager = capture == cudaStreamCaptureStatusNone;
  if (!search && lay.bytes > ctx->scratch_bytes && may_search_for_chunks(ctx, M, nnz, n_chunks) &&
      (!eager || hpspmm_try_scratch(ctx, lay.bytes) != HPSPMM_OK)) {
    search = true;
    lay = planless_layout(M, K, n_chunks, true);
  }
  st = hpspmm_ensure_scratch(ctx, lay.bytes);
  if (st == HPSPMM_OK && eager) st = hpspmm_ensure_counters(ctx, counters_to_keep(ctx, K, lay.n_counter, search), s);
  if (st != HPSPMM_OK) return st;
  char* base = (char*)ctx->scratch;
  a.n_chunks = (int)n_chunks, a.S = S;
  a.carry = (float*)(base + lay.carry), a.counter = (int32_t*)(base + lay.counter);
  // The counters of split rows have to be zero when the product starts.  Where the structure is built first, that clears
  // them.  A product of one launch takes them from sets of their own, cleared by the product before it (a memset in front
  // costs 2 us of a product of 8), unless the call is being captured.
  if (!search) {
    int4* rec = (int4*)(base + lay.rec);
    int2* nz = (int2*)(base + lay.nz);
    st = hpspmm_build_structure(ctx, M, nnz, row_ptr, S, n_chunks, nz, rec, (int32_t*)(base + lay.tiles),
                                hpspmm_structure_tables{}, s, a.counter, lay.n_counter);
    if (st != HPSPMM_OK) return st;
    a.rec = rec, a.nz = nz;
    return launch_spmm(ctx, a, hint, false, false, s);
  }
  if (!eager) {
    HPSPMM_CUDA_TRY(ctx, cudaMemsetAsync(a.counter, 0, (size_t)lay.n_counter * 4, s));
    return launch_spmm(ctx, a, hint, false, false, s);
  }
  hpspmm_take_counters(ctx, &a.counter, &a.clear, &a.n_clear);
  st = launch_spmm(ctx, a, hint, false, false, s);
  hpspmm_counters_used(ctx, lay.n_counter, st == HPSPMM_OK);
  return st;
}

// Host-buffer products, pipelined over column slabs: C[:, s] = A * B[:, s] needs only slab s of B,
// so slab s+1 is uploaded (strided 2-D copy) while slab s is multiplied (as a contiguous product of
// the slab's width) and slab s-1 is downloaded.  PCIe is full duplex: the downloads hide behind the
// uploads.  A is uploaded once, in front; the slabs of several products that share A follow one
// another through the same pipeline, so the whole call costs about
// upload(A) + upload(all B) + product and download of the last slab.
namespace {
struct host_slab {
  const float* B;   // host, first column of the slab
  float* C;         // host, first column of the slab
  int64_t K;        // row stride of the host matrices
  int64_t width;    // 32 or 64 (or K itself for widths that are not multiples of 32)
};
}  // namespace

static int host_products_pipelined(hpspmm_ctx* ctx, int64_t M, int64_t N, int64_t nnz, const int32_t* row_ptr,
                                   const int32_t* col_idx, const float* vals, const host_slab* slabs, int n_slabs,
                                   const hpspmm_opts* opts) {
  constexpr int NBUF = 2;
  for (int i = 0; i < 3; ++i)
    if (!ctx->pipe_streams[i])
      HPSPMM_CUDA_TRY(ctx, cudaStreamCreateWithFlags(&ctx->pipe_streams[i], cudaStreamNonBlocking));
  // the events live in the context: created once, never leaked by an error path of a call
  for (int i = 0; i < 1 + 3 * NBUF; ++i)
    if (!ctx->pipe_events[i])
      HPSPMM_CUDA_TRY(ctx, cudaEventCreateWithFlags(&ctx->pipe_events[i], cudaEventDisableTiming));
  cudaStream_t s_in = ctx->pipe_streams[0], s_run = ctx->pipe_streams[1], s_out = ctx->pipe_streams[2];
  cudaEvent_t ev_a = ctx->pipe_events[0];
  cudaEvent_t* ev_b = ctx->pipe_events + 1;
  cudaEvent_t* ev_run = ctx->pipe_events + 1 + NBUF;
  cudaEvent_t* ev_out = ctx->pipe_events + 1 + 2 * NBUF;
  int64_t wmax = 1;
  for (int i = 0; i < n_slabs; ++i) wmax = slabs[i].width > wmax ? slabs[i].width : wmax;
  const size_t b_rp = align_up((size_t)(M + 1) * 4, 256);
  const size_t b_nz = align_up((size_t)(nnz > 0 ? nnz : 1) * 4, 256);
  const size_t b_Bs = align_up((size_t)(N > 0 ? N : 1) * wmax * 4, 256);
  const size_t b_Cs = align_up((size_t)M * wmax * 4, 256);
  int st = hpspmm_ensure_stage(ctx, b_rp + 2 * b_nz + NBUF * (b_Bs + b_Cs));
  if (st != HPSPMM_OK) return st;
  // size the kernel scratch before anything is queued (growing it synchronises the device)
  {
    size_t need = 0, least = 0;   // least: with searches wherever they will do
    int64_t need_counters = 0;
    for (int i = 0; i < n_slabs; ++i) {
      const int64_t w = slabs[i].width;
      const int32_t S = planless_chunk_nnz(w, nnz, opts);
      const int64_t n_chunks = (nnz + S - 1) / S;
      const bool search = searches_for_chunks(ctx, M, w, nnz, n_chunks, S);
      const planless_layout lay(M, w, n_chunks, search);
      need = lay.bytes > need ? lay.bytes : need;
      const planless_layout small(M, w, n_chunks, search || may_search_for_chunks(ctx, M, nnz, n_chunks));
      least = small.bytes > least ? small.bytes : least;
      const int64_t keep = counters_to_keep(ctx, w, lay.n_counter, search);
      need_counters = keep > need_counters ? keep : need_counters;
    }
    if (least < need && hpspmm_try_scratch(ctx, need) != HPSPMM_OK) need = least;
    st = hpspmm_ensure_scratch(ctx, need);
    if (st == HPSPMM_OK) st = hpspmm_ensure_counters(ctx, need_counters, s_run);
    if (st != HPSPMM_OK) return st;
  }
  char* base = (char*)ctx->stage;
  int32_t* d_rp = (int32_t*)base;
  int32_t* d_col = (int32_t*)(base + b_rp);
  float* d_val = (float*)(base + b_rp + b_nz);
  float* d_Bs[NBUF];
  float* d_Cs[NBUF];
  for (int i = 0; i < NBUF; ++i) {
    d_Bs[i] = (float*)(base + b_rp + 2 * b_nz + i * b_Bs);
    d_Cs[i] = (float*)(base + b_rp + 2 * b_nz + NBUF * b_Bs + i * b_Cs);
  }
  int rc = HPSPMM_OK;
  cudaError_t e = cudaSuccess;
#define PIPE_TRY(call)                      \
  if (rc == HPSPMM_OK && e == cudaSuccess) { \
    e = (call);                             \
  }
  PIPE_TRY(cudaMemcpyAsync(d_rp, row_ptr, (size_t)(M + 1) * 4, cudaMemcpyHostToDevice, s_in));
  if (nnz > 0) {
    PIPE_TRY(cudaMemcpyAsync(d_col, col_idx, (size_t)nnz * 4, cudaMemcpyHostToDevice, s_in));
    PIPE_TRY(cudaMemcpyAsync(d_val, vals, (size_t)nnz * 4, cudaMemcpyHostToDevice, s_in));
  }
  PIPE_TRY(cudaEventRecord(ev_a, s_in));
  PIPE_TRY(cudaStreamWaitEvent(s_run, ev_a, 0));
  for (int s = 0; s < n_slabs; ++s) {
    const int buf = s % NBUF;
    const host_slab& sl = slabs[s];
    // upload slab s once the product that last read this buffer is done
    if (s >= NBUF) PIPE_TRY(cudaStreamWaitEvent(s_in, ev_run[buf], 0));
    if (nnz > 0 && N > 0)
      PIPE_TRY(cudaMemcpy2DAsync(d_Bs[buf], sl.width * 4, sl.B, (size_t)sl.K * 4, sl.width * 4, (size_t)N,
                                 cudaMemcpyHostToDevice, s_in));
    PIPE_TRY(cudaEventRecord(ev_b[buf], s_in));
    // multiply once the slab has landed and the previous download from this C buffer is done
    PIPE_TRY(cudaStreamWaitEvent(s_run, ev_b[buf], 0));
    if (s >= NBUF) PIPE_TRY(cudaStreamWaitEvent(s_run, ev_out[buf], 0));
    if (rc == HPSPMM_OK && e == cudaSuccess)
      rc = hpspmm_spmm_csr_f32(ctx, nullptr, M, N, sl.width, nnz, d_rp, d_col, d_val, d_Bs[buf], d_Cs[buf], opts,
                               (hpspmm_stream)s_run);
    PIPE_TRY(cudaEventRecord(ev_run[buf], s_run));
    // download
    PIPE_TRY(cudaStreamWaitEvent(s_out, ev_run[buf], 0));
    PIPE_TRY(cudaMemcpy2DAsync(sl.C, (size_t)sl.K * 4, d_Cs[buf], sl.width * 4, sl.width * 4, (size_t)M,
                               cudaMemcpyDeviceToHost, s_out));
    PIPE_TRY(cudaEventRecord(ev_out[buf], s_out));
  }
#undef PIPE_TRY
  // drain all three streams whatever happened
  cudaError_t e1 = cudaStreamSynchronize(s_in), e2 = cudaStreamSynchronize(s_run), e3 = cudaStreamSynchronize(s_out);
  if (rc != HPSPMM_OK) return rc;
  if (e == cudaSuccess) e = e1 != cudaSuccess ? e1 : (e2 != cudaSuccess ? e2 : e3);
  if (e != cudaSuccess) return hpspmm_set_err(ctx, HPSPMM_ERR_CUDA, "host-buffer product pipeline", e);
  return HPSPMM_OK;
}

// The same for operands so small that issuing the pipeline takes longer than the copies it overlaps: whole products,
// one stream, one synchronisation.  slabs[i] are whole products (width == K).
static int host_products_in_turn(hpspmm_ctx* ctx, int64_t M, int64_t N, int64_t nnz, const int32_t* row_ptr,
                                 const int32_t* col_idx, const float* vals, const host_slab* slabs, int n_slabs,
                                 const hpspmm_opts* opts, cudaStream_t s) {
  int64_t wmax = 1;
  for (int i = 0; i < n_slabs; ++i) wmax = slabs[i].width > wmax ? slabs[i].width : wmax;
  const size_t b_rp = align_up((size_t)(M + 1) * 4, 256);
  const size_t b_nz = align_up((size_t)(nnz > 0 ? nnz : 1) * 4, 256);
  const size_t b_B = align_up((size_t)(N > 0 ? N : 1) * wmax * 4, 256);
  int st = hpspmm_ensure_stage(ctx, b_rp + 2 * b_nz + b_B + (size_t)M * wmax * 4);
  if (st != HPSPMM_OK) return st;
  char* base = (char*)ctx->stage;
  int32_t* d_rp = (int32_t*)base;
  int32_t* d_col = (int32_t*)(base + b_rp);
  float* d_val = (float*)(base + b_rp + b_nz);
  float* d_B = (float*)(base + b_rp + 2 * b_nz);
  float* d_C = (float*)(base + b_rp + 2 * b_nz + b_B);
  cudaError_t e = cudaMemcpyAsync(d_rp, row_ptr, (size_t)(M + 1) * 4, cudaMemcpyHostToDevice, s);
  if (nnz > 0) {
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_col, col_idx, (size_t)nnz * 4, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_val, vals, (size_t)nnz * 4, cudaMemcpyHostToDevice, s);
  }
  for (int i = 0; i < n_slabs && e == cudaSuccess && st == HPSPMM_OK; ++i) {
    const host_slab& p = slabs[i];
    if (nnz > 0 && N > 0) e = cudaMemcpyAsync(d_B, p.B, (size_t)N * p.K * 4, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess)
      st = hpspmm_spmm_csr_f32(ctx, nullptr, M, N, p.K, nnz, d_rp, d_col, d_val, d_B, d_C, opts, (hpspmm_stream)s);
    if (e == cudaSuccess && st == HPSPMM_OK)
      e = cudaMemcpyAsync(p.C, d_C, (size_t)M * p.K * 4, cudaMemcpyDeviceToHost, s);
  }
  const cudaError_t e1 = cudaStreamSynchronize(s);   // whatever happened
  if (st != HPSPMM_OK) return st;
  if (e == cudaSuccess) e = e1;
  if (e != cudaSuccess) return hpspmm_set_err(ctx, HPSPMM_ERR_CUDA, "host-buffer products", e);
  return HPSPMM_OK;
}

static int first_pipe_stream(hpspmm_ctx* ctx) {   // the device is current
  if (!ctx->pipe_streams[0])
    HPSPMM_CUDA_TRY(ctx, cudaStreamCreateWithFlags(&ctx->pipe_streams[0], cudaStreamNonBlocking));
  return HPSPMM_OK;
}

// Up to here the dense operands travel whole, one after the other: at 55 GB/s they take 75 us, and a slab of the
// pipeline costs about 15 us to issue.
static const int64_t kHostInTurnBytes = 4 << 20;

// Width of the column slabs a product of width K travels in.  64 columns when they divide K and leave at
// least two slabs: with both directions busy this link moves 256-byte rows at 50 GB/s each way and 128-byte
// rows at 36.  `others_overlap` (several products in one call): a 64-column product then travels whole, as
// one contiguous copy, and overlaps with its neighbours instead of with itself.  Else 32; a width that is
// no multiple of 32 travels whole.
static int64_t host_slab_width(int64_t K, bool others_overlap) {
  if (K % 32 != 0) return K;
  return (K % 64 == 0 && (K >= 128 || others_overlap)) ? 64 : 32;
}

static int append_slabs(host_slab* out, int cap, int n, const float* B, float* C, int64_t K,
                        bool others_overlap = false) {
  if (K % 32 != 0) {
    if (n >= cap) return -1;
    out[n++] = host_slab{B, C, K, K};
    return n;
  }
  const int64_t w = host_slab_width(K, others_overlap);
  for (int64_t off = 0; off < K; off += w) {
    if (n >= cap) return -1;
    out[n++] = host_slab{B + off, C + off, K, w};
  }
  return n;
}

static int host_product_slabs(hpspmm_ctx* ctx, int64_t M, int64_t N, int64_t K, int64_t nnz,
                              const int32_t* row_ptr, const int32_t* col_idx, const float* vals,
                              const float* B, float* C, const hpspmm_opts* opts) {
  host_slab slabs[64];
  const int n = append_slabs(slabs, 64, 0, B, C, K);
  if (n < 0) return HPSPMM_ERR_UNSUPPORTED;
  return host_products_pipelined(ctx, M, N, nnz, row_ptr, col_idx, vals, slabs, n, opts);
}

int hpspmm_spmm_csr_f32_host_multi(hpspmm_ctx* ctx, int64_t M, int64_t N, int64_t nnz, const int32_t* row_ptr,
                                   const int32_t* col_idx, const float* vals, int32_t n_products, const int64_t* Ks,
                                   const float* const* Bs, float* const* Cs, const hpspmm_opts* opts) {
  HPSPMM_TRACE("hpspmm_spmm_csr_f32_host_multi");
  HPSPMM_REQUIRE(ctx, ctx != nullptr, "null context");
  HPSPMM_REQUIRE(ctx, M >= 0 && N >= 0 && nnz >= 0, "bad size");
  HPSPMM_REQUIRE(ctx, n_products >= 0 && n_products <= 16, "between 0 and 16 products per call");
  HPSPMM_REQUIRE(ctx, n_products == 0 || (Ks && Bs && Cs), "null product list");
  HPSPMM_REQUIRE(ctx, row_ptr != nullptr, "null row_ptr");
  HPSPMM_REQUIRE(ctx, nnz == 0 || (col_idx && vals), "null operand");
  if (M == 0 || n_products == 0) return HPSPMM_OK;
  const int algo = opts ? opts->algo : HPSPMM_ALGO_AUTO;
  HPSPMM_REQUIRE(ctx, algo != HPSPMM_ALGO_ROW_SPLIT, "the multi-product entry runs the balanced kernels only");
  host_slab slabs[16 * 16];
  int n = 0;
  for (int i = 0; i < n_products; ++i) {
    HPSPMM_REQUIRE(ctx, Ks[i] >= 1 && Ks[i] <= 512, "K must be between 1 and 512");
    HPSPMM_REQUIRE(ctx, Cs[i] != nullptr && (nnz == 0 || Bs[i] != nullptr), "null dense operand");
  }
  int64_t dense = 0;
  for (int i = 0; i < n_products; ++i) dense += 4 * Ks[i] * (M + N);
  if (dense <= kHostInTurnBytes) {
    for (int i = 0; i < n_products; ++i) slabs[i] = host_slab{Bs[i], Cs[i], Ks[i], Ks[i]};
    hpspmm_device_guard guard(ctx->device);
    const int st = first_pipe_stream(ctx);
    if (st != HPSPMM_OK) return st;
    return host_products_in_turn(ctx, M, N, nnz, row_ptr, col_idx, vals, slabs, n_products, opts, ctx->pipe_streams[0]);
  }
  // Order of the products.  Downloads can start only after the first slab has been uploaded and multiplied, and the
  // download of the very last slab overlaps nothing, so the pipeline should begin AND end on a narrow slab: the
  // product with the narrowest slabs goes last, the next narrowest first, the others between them, widest first.
  const bool several = n_products >= 2;
  auto slab_width = [&](int i) { return host_slab_width(Ks[i], several); };
  int order[16];
  for (int i = 0; i < n_products; ++i) order[i] = i;
  std::stable_sort(order, order + n_products, [&](int a, int b) {
    return slab_width(a) != slab_width(b) ? slab_width(a) > slab_width(b) : Ks[a] > Ks[b];
  });
  if (n_products >= 3) {
    // order is now widest .. narrowest; bring the second narrowest to the front
    const int second = order[n_products - 2];
    for (int i = n_products - 2; i > 0; --i) order[i] = order[i - 1];
    order[0] = second;
  }
  for (int i = 0; i < n_products; ++i) {
    n = append_slabs(slabs, 16 * 16, n, Bs[order[i]], Cs[order[i]], Ks[order[i]], several);
    if (n < 0) return HPSPMM_ERR_UNSUPPORTED;
  }
  hpspmm_device_guard guard(ctx->device);
  return host_products_pipelined(ctx, M, N, nnz, row_ptr, col_idx, vals, slabs, n, opts);
}

int hpspmm_spmm_csr_f32_host(hpspmm_ctx* ctx, int64_t M, int64_t N, int64_t K, int64_t nnz,
                             const int32_t* row_ptr, const int32_t* col_idx, const float* vals,
                             const float* B, float* C, const hpspmm_opts* opts) {
  HPSPMM_TRACE("hpspmm_spmm_csr_f32_host");
  HPSPMM_REQUIRE(ctx, ctx != nullptr, "null context");
  HPSPMM_REQUIRE(ctx, M >= 0 && N >= 0 && nnz >= 0 && K >= 1, "bad size");
  HPSPMM_REQUIRE(ctx, row_ptr != nullptr, "null row_ptr");
  HPSPMM_REQUIRE(ctx, nnz == 0 || (col_idx && vals && B), "null operand");
  HPSPMM_REQUIRE(ctx, M == 0 || C != nullptr, "null output");
  if (M == 0) return HPSPMM_OK;
  hpspmm_device_guard guard(ctx->device);
  int st = HPSPMM_OK;
  const int algo = opts ? opts->algo : HPSPMM_ALGO_AUTO;
  const host_slab whole = {B, C, K, K};
  if (nnz > 0 && N > 0 && K >= 64 && K % 32 == 0 && algo != HPSPMM_ALGO_ROW_SPLIT) {
    if (4 * K * (M + N) > kHostInTurnBytes)
      return host_product_slabs(ctx, M, N, K, nnz, row_ptr, col_idx, vals, B, C, opts);
    // these widths run beside the default stream, whatever their size
    if ((st = first_pipe_stream(ctx)) != HPSPMM_OK) return st;
    return host_products_in_turn(ctx, M, N, nnz, row_ptr, col_idx, vals, &whole, 1, opts, ctx->pipe_streams[0]);
  }
  return host_products_in_turn(ctx, M, N, nnz, row_ptr, col_idx, vals, &whole, 1, opts, /*default stream*/ 0);
}

}  // extern "C"

// ---- CSR SpMM with its scratch in a static device array -----------------------------------
// Some callers must not allocate device memory at the moment they need a product: the
// enqueue hook of an inference-runtime plugin, a step inside a serving loop whose framework
// allocator already owns every byte of the device, or code on a latency budget that cannot
// afford the device-wide synchronisation an allocation may cause.  For them the chunk table
// and the carry slots live in the array below instead of in context-owned scratch.  The
// array is part of the library image: every GPU that loads the library holds these bytes
// until the process exits, which is why the limit is modest.
#define HPSPMM_STATIC_SCRATCH_BYTES (16u << 20)
static __device__ __align__(256) unsigned char g_static_scratch[HPSPMM_STATIC_SCRATCH_BYTES];

namespace {

constexpr int kMaxStaticDevices = 64;
struct static_scratch_state {
  bool ready;
  unsigned char* base;  // device address of g_static_scratch on this device
  int sm_count;
};
static_scratch_state g_static_state[kMaxStaticDevices];
std::mutex g_static_mutex;

void write_err(char* buf, size_t len, const char* msg) {
  if (buf && len) snprintf(buf, len, "%s", msg);
}

}  // namespace

extern "C" int hpspmm_spmm_csr_f32_static_scratch(int device_ordinal, int64_t M, int64_t N,
                                                  int64_t K, int64_t nnz, const int32_t* row_ptr,
                                                  const int32_t* col_idx, const float* vals,
                                                  const float* B, float* C, hpspmm_stream stream,
                                                  char* err_buf, size_t err_len) {
  if (err_buf && err_len) err_buf[0] = 0;
  if (device_ordinal < 0 || device_ordinal >= kMaxStaticDevices) {
    write_err(err_buf, err_len, "device ordinal out of range");
    return HPSPMM_ERR_INVALID;
  }
  {
    // a device the process cannot see must be refused here: making it current below would fail
    // silently and the array's address would be looked up on whichever device happens to be current
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || device_ordinal >= count) {
      char msg[128];
      snprintf(msg, sizeof(msg), "device ordinal %d does not exist (%d visible)", device_ordinal, count);
      write_err(err_buf, err_len, msg);
      return HPSPMM_ERR_INVALID;
    }
  }
  hpspmm_ctx local;  // a stack stand-in for a context: no allocation behind it
  memset(&local, 0, sizeof(local));
  local.device = device_ordinal;
  int st = check_spmm_args(&local, M, N, K, nnz, row_ptr, col_idx, vals, B, C);
  if (st != HPSPMM_OK) {
    write_err(err_buf, err_len, local.err);
    return st;
  }
  if (M == 0) return HPSPMM_OK;

  // small matrices take the (smaller) chunks of the ordinary entry point where they fit
  int32_t S = hpspmm_default_chunk_nnz(K, nnz);
  int64_t n_chunks;
  size_t b_int, need;
  for (;;) {
    if (S > probing_chunk_nnz(K)) S = probing_chunk_nnz(K);
    n_chunks = (nnz + S - 1) / S;
    b_int = align_up((size_t)(n_chunks + 1) * 4, 256);
    need = b_int + align_up((size_t)(n_chunks + 1) * (size_t)K * 4, 256);
    if (need <= (size_t)HPSPMM_STATIC_SCRATCH_BYTES || S == probing_chunk_nnz(K)) break;
    S = probing_chunk_nnz(K);
  }
  if (need > (size_t)HPSPMM_STATIC_SCRATCH_BYTES) {
    char msg[256];
    const long long max_chunks = (long long)(HPSPMM_STATIC_SCRATCH_BYTES - 2 * 256) / (4 + 4 * K) - 1;
    snprintf(msg, sizeof(msg),
             "matrix too large for the static scratch: nnz = %lld at K = %lld needs %zu bytes, the "
             "array holds %u (about %lld nnz at this K); use hpspmm_spmm_csr_f32 instead",
             (long long)nnz, (long long)K, need, (unsigned)HPSPMM_STATIC_SCRATCH_BYTES,
             max_chunks > 0 ? max_chunks * S : 0ll);
    write_err(err_buf, err_len, msg);
    return HPSPMM_ERR_UNSUPPORTED;
  }

  hpspmm_device_guard guard(device_ordinal);  // the device is current from here on
  static_scratch_state& state = g_static_state[device_ordinal];
  {
    // Once per device: the array's name is a host-side handle, not a device address, so ask
    // the runtime where the array lives on the current device.
    std::lock_guard<std::mutex> lock(g_static_mutex);
    if (!state.ready) {
      void* p = nullptr;
      cudaError_t e = cudaGetSymbolAddress(&p, g_static_scratch);
      if (e != cudaSuccess || p == nullptr) {
        char msg[200];
        snprintf(msg, sizeof(msg), "cudaGetSymbolAddress(static scratch): %s", cudaGetErrorString(e));
        write_err(err_buf, err_len, msg);
        return HPSPMM_ERR_CUDA;
      }
      int sms = 0;
      e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device_ordinal);
      if (e != cudaSuccess || sms <= 0) {
        write_err(err_buf, err_len, "cudaDeviceGetAttribute(multiprocessor count) failed");
        return HPSPMM_ERR_CUDA;
      }
      state.base = (unsigned char*)p;
      state.sm_count = sms;
      state.ready = true;
    }
  }
  local.sm_count = state.sm_count;

  // Every call zeroes the per-row counters, and a carry slot is read only where this call hands a carry on, so
  // nothing left over from an earlier call is ever consumed.
  int32_t* run_counter = (int32_t*)state.base;
  cudaStream_t s = (cudaStream_t)stream;
  cudaError_t e = cudaMemsetAsync(run_counter, 0, b_int, s);
  if (e != cudaSuccess) {
    write_err(err_buf, err_len, cudaGetErrorString(e));
    return HPSPMM_ERR_CUDA;
  }
  hpspmm_spmm_args a;
  memset(&a, 0, sizeof(a));
  a.M = (int)M, a.K = (int)K, a.n_chunks = (int)n_chunks, a.S = S;
  a.row_ptr = row_ptr, a.col_idx = col_idx, a.vals = vals, a.B = B, a.C = C;
  a.carry = (float*)(state.base + b_int), a.counter = run_counter;
  st = launch_spmm(&local, a, gather_hint(K, nullptr), /*even=*/false, /*shared_counters=*/true, s);
  if (st != HPSPMM_OK) write_err(err_buf, err_len, local.err);
  return st;
}

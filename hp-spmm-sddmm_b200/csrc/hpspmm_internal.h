// Internal declarations shared by the translation units of libhpspmm.so.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include "hpspmm.h"

// Context: device ordinal, cached device properties, grow-only scratch and the text
// of the last CUDA error.  Takes the place of starml's allocator and handle
// registries (spmm/starml/basic/allocator.cpp:21-48, spmm/starml/basic/handle.cpp:11-17).
struct hpspmm_ctx {
  int device;
  int sm_count;
  int64_t l2_bytes;
  int max_smem_optin;
  int64_t launches;
  // scratch for plan-less calls: chunk table and carries
  void* scratch;
  size_t scratch_bytes;
  // split-row counters of plan-less products that run as one launch: two sets of counter_cap ints in a block that
  // nothing else writes.  A product counts in one set and clears what the one before it may have left in the other
  // (hpspmm_take_counters).
  int32_t* counters;
  int64_t counter_cap;
  int64_t counter_used[2];
  int counter_turn;
  bool counters_unknown;   // a launch failed between the two: both sets are cleared before the next use
  // staging for the host-buffer entry point
  void* stage;
  size_t stage_bytes;
  int* flag;  // 64 device ints: [0] validation and plan building, [HPSPMM_FLAG_TMA_FALLBACKS] see below
  // streams of the host-buffer entry point: uploads, kernels, downloads (created on first use)
  cudaStream_t pipe_streams[3];
  cudaEvent_t pipe_events[8];   // "A has landed" and, per buffer, slab uploaded / multiplied / downloaded
  char err[256];
};

// ctx->flag[HPSPMM_FLAG_TMA_FALLBACKS] counts the warps of spmm_tma_kernel whose bounded wait for a TMA copy
// ran out (they finish their chunk with ordinary loads); hpspmm_ctx_tma_fallbacks reads it.
#define HPSPMM_FLAG_TMA_FALLBACKS 16

// Chunk table of one sparsity structure.
//   chunk_start[c]  first nnz of chunk c (n_chunks + 1 entries)
//   chunk_row[c]    row holding nnz chunk_start[c]
//   carry_val[c*K..] partial sum of a row that chunk c hands on
//   rec             the same per chunk in the order in which warps take them, see hpspmm_spmm_args
struct hpspmm_plan {
  int device;
  int sm_count;
  int64_t M, nnz;
  int32_t chunk_nnz;
  int64_t n_chunks;
  int64_t n_split_chunks;  // chunks that end inside a row
  int64_t max_K;
  int32_t* chunk_start;
  int32_t* chunk_row;
  int32_t* chunk_order;  // chunk ids, most rows first: the order in which warps take chunks
  float* carry_val;
  int32_t* run_counter;  // hpspmm_counter_slabs(max_K) per chunk, zero between launches: pieces of a split row that have finished
  // rows that hold entries: ids (ascending, then the sentinel M), their ends in the entry array, and
  // for every chunk the position in this list of the row holding its first entry
  int32_t* nz_id;
  int32_t* nz_end;
  int32_t* chunk_ri;
  int2* nz;        // (nz_id, nz_end) as one word per row: what the product kernels step through
  int4* rec;
  size_t bytes;
};

// Whether the rows of the plan's matrix are of even length: few of them are longer than a chunk.  A power-law graph has
// a chunk in two to a chunk in four beginning inside a row, uniform rows have none.
static inline bool hpspmm_even_rows(const hpspmm_plan* p) { return p->n_split_chunks * 8 < p->n_chunks; }

// What the CSR product kernels are launched with.
//   rec, 32 bytes per slot of the schedule: {n0, ri, row, row_end} {chunk, row_start, n1, -}: entries [n0, n1) of the
//   chunk, the row holding entry n0 with its bounds and its position in the list of rows.  One aligned load gives a
//   warp all it needs, where chunk_order -> chunk_start / chunk_ri -> nz_id are three dependent ones.
//   rec and nz null: warps take the chunks in matrix order, search row_ptr for their bounds and step along row_ptr.
struct hpspmm_spmm_args {
  int M, K, n_chunks, S;
  int off, cols;               // columns of this launch: [off, off + cols), in slabs of the shape's width
  int n_chunk_blocks, slab0;   // filled in by the launcher
  int keep_b;                  // L2 evict-last on the gathers of B
  const int32_t* row_ptr;
  const int32_t* col_idx;
  const float* vals;
  const float* B;
  float* C;
  const int4* rec;
  const int2* nz;
  float* carry;
  int32_t* counter;
  int32_t* clear;   // n_clear ints that the kernel without a list sets to zero, for the next product (hpspmm_take_counters)
  int n_clear;
};
// Shape of the kernel for `cols` columns: VEC-wide vectors, W lanes and R vectors per lane to a group (warp_frag.cuh).
struct hpspmm_spmm_shape {
  int VEC, W, R;
  bool lat;    // few chunks: more gathers in flight per warp
  bool mid;    // one or two waves of 24 warps per SM: twice the gathers in flight (wide groups of 16-byte vectors)
  bool hint;
};
// widest vector the rows of the dense operands keep aligned; addresses: bitwise or of the operands' addresses
int hpspmm_vector_width(int64_t K, uintptr_t addresses);
hpspmm_spmm_shape hpspmm_choose_shape(int VEC, int64_t cols, int widest, bool hint);
// Widest slab one shape covers (four vectors per lane, eight of 4 bytes).  A wider product runs as that many full
// slabs and one launch for the rest, so that only the last vector of a lane can ever lie outside a slab.
static inline int hpspmm_widest_slab(int VEC) { return VEC == 1 ? 256 : 128 * VEC; }
// The kernels rely on that: every slab of `cols` columns reaches into the last vector of its lanes.
static inline bool hpspmm_shape_covers(int VEC, int W, int R, int cols) {
  const int cw = VEC * W * R, last = cols % cw == 0 ? cw : cols % cw;
  return cols > 0 && last > VEC * W * (R - 1);
}
static inline int hpspmm_launch_cols(int K, int off, int widest) {
  const int left = K - off;
  return left < widest ? left : left / widest * widest;
}
// triples per warp of the COO product
int32_t hpspmm_coo_chunk_nnz(int64_t K, int64_t nnz);
int hpspmm_spmm_launch_v4(hpspmm_ctx* ctx, const hpspmm_spmm_args& a, const hpspmm_spmm_shape& sh, bool shared_counters,
                          cudaStream_t s);
int hpspmm_spmm_launch_v2(hpspmm_ctx* ctx, const hpspmm_spmm_args& a, const hpspmm_spmm_shape& sh, bool shared_counters,
                          cudaStream_t s);
int hpspmm_spmm_launch_v1(hpspmm_ctx* ctx, const hpspmm_spmm_args& a, const hpspmm_spmm_shape& sh, bool shared_counters,
                          cudaStream_t s);
// sets of per-chunk counters a product of up to K columns may need: one per slab, no slab narrower than 32 columns
static inline int64_t hpspmm_counter_slabs(int64_t K) { return (K + 31) / 32; }

// What the kernel of both layer gradients is launched with: the transpose of A by rows (row_ptr, col_idx, and perm, the
// position of every entry in A's order) with its plan's tables, and the dense operands, K columns wide.
struct hpspmm_layer_grad_args {
  int rows, K, n_chunks, S;
  int n_chunk_blocks;   // filled in by the launcher
  int keep;             // L2 evict-last on the gathers of dC
  const int32_t* row_ptr;
  const int32_t* col_idx;
  const int32_t* perm;
  const float* vals;    // weights in A's order
  const float* dC;
  const float* H;
  float* dH;
  float* dA;
  const int4* rec;
  const int2* nz;
  float* carry;
  int32_t* counter;
};
// whether the kernel has a shape for K columns at these operands (addresses: or of theirs)
bool hpspmm_layer_grad_covers(int64_t K, uintptr_t addresses);
// whether the one kernel beats the three it replaces; M: rows of dC, VEC: hpspmm_vector_width of the operands, even: rows of
// even length (hpspmm_even_rows), captured: the call is recorded in a graph
bool hpspmm_layer_grad_pays(const hpspmm_ctx* ctx, int64_t M, int64_t K, int VEC, int64_t nnz, bool even, bool captured);
int hpspmm_layer_grad_launch(hpspmm_ctx* ctx, const hpspmm_layer_grad_args& a, cudaStream_t s);

static inline int hpspmm_set_err(hpspmm_ctx* ctx, int status, const char* what, cudaError_t e) {
  if (ctx) snprintf(ctx->err, sizeof(ctx->err), "%s: %s", what, cudaGetErrorString(e));
  return status;
}

#define HPSPMM_CUDA_TRY(ctx, call)                                               \
  do {                                                                           \
    cudaError_t e__ = (call);                                                    \
    if (e__ != cudaSuccess)                                                      \
      return hpspmm_set_err((ctx), e__ == cudaErrorMemoryAllocation ? HPSPMM_ERR_OOM \
                                                                   : HPSPMM_ERR_CUDA, \
                            #call, e__);                                         \
  } while (0)

#define HPSPMM_REQUIRE(ctx, cond, msg)                                     \
  do {                                                                     \
    if (!(cond)) {                                                         \
      if (ctx) snprintf((ctx)->err, sizeof((ctx)->err), "invalid argument: %s", msg); \
      return HPSPMM_ERR_INVALID;                                           \
    }                                                                      \
  } while (0)

// Makes the context's device current for the calling thread for the duration of a call.
struct hpspmm_device_guard {
  int prev;
  bool switched;
  explicit hpspmm_device_guard(int dev) : prev(-1), switched(false) {
    if (cudaGetDevice(&prev) == cudaSuccess && prev != dev) {
      cudaSetDevice(dev);
      switched = true;
    }
  }
  ~hpspmm_device_guard() {
    if (switched) cudaSetDevice(prev);
  }
};

// Every device allocation of the library goes through here: cudaMalloc, unless a test has armed
// hpspmm_debug_fail_device_alloc, in which case the chosen allocation reports cudaErrorMemoryAllocation
// without touching the device.
cudaError_t hpspmm_device_malloc(void** out, size_t bytes);
template <typename T>
static inline cudaError_t hpspmm_device_malloc(T** out, size_t bytes) {
  return hpspmm_device_malloc(reinterpret_cast<void**>(out), bytes);
}

// A named range around an entry point for timeline tools (NVTX 3, header-only: nothing to link, and a call is a
// null-pointer test when no tool is attached).  The reference has no tracing beyond its event timer
// (include/spmm/utils/timer_cuda.h:6-40).
#include <nvtx3/nvToolsExt.h>
struct hpspmm_trace_range {
  explicit hpspmm_trace_range(const char* name) { nvtxRangePushA(name); }
  ~hpspmm_trace_range() { nvtxRangePop(); }
  hpspmm_trace_range(const hpspmm_trace_range&) = delete;
  hpspmm_trace_range& operator=(const hpspmm_trace_range&) = delete;
};
#define HPSPMM_TRACE(name) hpspmm_trace_range hpspmm_trace_range__(name)

int hpspmm_ensure_scratch(hpspmm_ctx* ctx, size_t bytes);
// the same for a caller that can do with less: HPSPMM_ERR_OOM leaves the scratch as it was
int hpspmm_try_scratch(hpspmm_ctx* ctx, size_t bytes);
// Two sets of at least `n` counters, zero when work queued on `stream` starts.  hpspmm_take_counters hands out the set for
// one product, whose kernel clears the first `*n_clear` ints at `*clear`; hpspmm_counters_used tells how many it counts in
// and how its launch went.  Not for captured calls: a graph may be replayed between any two products, so a captured call
// keeps its counters in the scratch and clears them itself.
int hpspmm_ensure_counters(hpspmm_ctx* ctx, int64_t n, cudaStream_t stream);
void hpspmm_take_counters(hpspmm_ctx* ctx, int32_t** set, int32_t** clear, int* n_clear);
void hpspmm_counters_used(hpspmm_ctx* ctx, int64_t n, bool launched);
int hpspmm_ensure_stage(hpspmm_ctx* ctx, size_t bytes);

// nominal chunk size for a dense width and a matrix of nnz entries
int32_t hpspmm_default_chunk_nnz(int64_t K, int64_t nnz);

// Processing order of the chunks: chunk ids sorted by estimated cost (entries / 8 + rows / 2),
// most expensive first (stable 8-bit counting-sort passes on the device).  Chunks full of short
// rows started last leave the GPU draining; started first they overlap with the others.
// With col_idx (may be null) the chunks that lie inside one row come last, in ascending order
// of their first column, so that pieces of different heavy rows running together read the same
// band of B.  `scratch` needs hpspmm_order_scratch_bytes(n_chunks) bytes.
size_t hpspmm_order_scratch_bytes(int64_t n_chunks);
int hpspmm_order_chunks_by_cost(hpspmm_ctx* ctx, int64_t M, int64_t N, int64_t n_chunks,
                                const int32_t* row_ptr, const int32_t* col_idx, const int32_t* chunk_start,
                                const int32_t* chunk_row, int32_t* order_out, void* scratch,
                                cudaStream_t stream);

// Builds the structure a product walks, in two launches: the list of rows that hold entries (nz, hpspmm_nz_bytes(M)
// bytes, with sentinels (M, INT_MAX) at its end) and one record per chunk (rec_out, 2 * n_chunks int4): in matrix order with
// `tables`, without them the chunks that lie inside one row after all others.
// counts: hpspmm_row_tile_ints(M) ints of scratch.  The first launch also sets `n_clear` ints at `clear` to zero.  The arrays of `tables` are
// filled as well where they are given (a plan exposes them), and split_count receives the number of chunks that
// begin inside a row.
struct hpspmm_structure_tables {
  int32_t* chunk_start;
  int32_t* chunk_row;
  int32_t* chunk_ri;
  int32_t* nz_id;
  int32_t* nz_end;
  int* split_count;
};
int64_t hpspmm_row_tile_ints(int64_t M);
size_t hpspmm_nz_bytes(int64_t M);
int hpspmm_build_structure(hpspmm_ctx* ctx, int64_t M, int64_t nnz, const int32_t* row_ptr, int32_t S, int64_t n_chunks,
                           int2* nz, int4* rec_out, int32_t* counts, const hpspmm_structure_tables& tables, cudaStream_t stream,
                           int32_t* clear = nullptr, int64_t n_clear = 0);
// rec[slot] = rec_in[order[slot]]
int hpspmm_order_records(hpspmm_ctx* ctx, int64_t n_chunks, const int32_t* order, const int4* rec_in, int4* rec,
                         cudaStream_t stream);

#if defined(__CUDACC__)
// Launches a kernel whose blocks may be set up before the kernel in front of it in the stream has ended (programmatic
// stream serialisation).  The kernel begins with chain_grid() (device_utils.cuh), so it touches no memory earlier than an
// ordinary launch would; what is saved is the time from the end of one kernel to the first instruction of the next.
// Passes back to back, ordinary launches -> these, us: product of 67.6 K entries, K = 32 10.6 -> 9.4, 1 M, K = 32 16.8 -> 14.4;
// without a plan 300 K, K = 100 24.3 -> 22.2, 1 M, K = 32 (three launches) 25.0 -> 18.8, 4 M, K = 64 101.2 -> 95.9; SDDMM of
// 100 K entries, K = 64 9.4 -> 7.8, 280 K, K = 160 18.9 -> 16.5; COO product of 280 K, K = 160 with its fill 20.9 -> 17.2.
template <typename... P, typename... A>
static inline void hpspmm_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = grid, c.blockDim = block, c.dynamicSmemBytes = smem, c.stream = s, c.attrs = &attr, c.numAttrs = 1;
  cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);   // (the caller asks cudaGetLastError)
}
#endif

// ---- counter-based PRNG shared by host and device --------------------------------------
// splitmix64 finaliser over (seed, stream, index); 24 high bits -> [0, 1).
#if defined(__CUDACC__)
#define HPSPMM_HD __host__ __device__ __forceinline__
#else
#define HPSPMM_HD static inline
#endif

HPSPMM_HD uint64_t hpspmm_mix64(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

HPSPMM_HD uint64_t hpspmm_rand64(uint64_t seed, uint64_t stream, uint64_t index) {
  uint64_t k = hpspmm_mix64(seed * 0x9E3779B97F4A7C15ull + stream + 0x632BE59BD9B4E019ull);
  return hpspmm_mix64(k + index * 0x9E3779B97F4A7C15ull);
}

// u in [0,1) on a 2^-24 grid: exact in fp32, so host and device agree bit for bit.
HPSPMM_HD float hpspmm_u01(uint64_t bits) { return (float)(uint32_t)(bits >> 40) * (1.0f / 16777216.0f); }

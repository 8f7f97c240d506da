// Register fragments of dense rows, as the warp kernels of the products gather, combine and store them.
//
// A warp is G = 32 / W lane groups of W lanes.  A group covers a slab of CW = VEC * W * R columns of a dense
// row: lane l of the group owns columns (r * W + l) * VEC .. + VEC - 1 for r < R.  VEC is the widest vector the
// row stride keeps aligned (K % 4 == 0: 16-byte loads, K even: 8-byte, K odd: 4-byte), W and R are the smallest
// that cover the slab.  A slab may be narrower than CW: a lane beyond its width kw gathers the slab's last vector
// instead (a line its neighbours read anyway, so no extra traffic and no predicate in the hot loop) and stores nothing.
#pragma once
#include "device_utils.cuh"

namespace hpspmm {

// one vector of a gathered row; HINT attaches an L2 eviction policy
template <int VEC, bool HINT>
__device__ __forceinline__ void gather_vec(float (&d)[VEC], const float* p, uint64_t policy) {
  if (VEC == 4) {
    const float4 v = ld_gather<HINT>(p, policy);
    d[0] = v.x, d[VEC > 1 ? 1 : 0] = v.y, d[VEC > 2 ? 2 : 0] = v.z, d[VEC > 3 ? 3 : 0] = v.w;
  } else if (VEC == 2) {
    if (HINT)
      asm("ld.global.nc.L2::cache_hint.v2.f32 {%0,%1}, [%2], %3;"
          : "=f"(d[0]), "=f"(d[VEC > 1 ? 1 : 0])
          : "l"(p), "l"(policy));
    else {
      const float2 v = __ldg(reinterpret_cast<const float2*>(p));
      d[0] = v.x, d[VEC > 1 ? 1 : 0] = v.y;
    }
  } else {
    if (HINT)
      asm("ld.global.nc.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(d[0]) : "l"(p), "l"(policy));
    else
      d[0] = __ldg(p);
  }
}

template <int N>
__device__ __forceinline__ void store_stream(float* p, const float (&v)[N]) {
  if (N == 4)
    st_stream(p, make_float4(v[0], v[N > 1 ? 1 : 0], v[N > 2 ? 2 : 0], v[N > 3 ? 3 : 0]));
  else if (N == 2)
    asm volatile("st.global.cs.v2.f32 [%0], {%1,%2};" ::"l"(p), "f"(v[0]), "f"(v[N > 1 ? 1 : 0]) : "memory");
  else
    asm volatile("st.global.cs.f32 [%0], %1;" ::"l"(p), "f"(v[0]) : "memory");
}

template <int N>
__device__ __forceinline__ void store_plain(float* p, const float (&v)[N]) {
  if (N == 4)
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[N > 1 ? 1 : 0], v[N > 2 ? 2 : 0], v[N > 3 ? 3 : 0]);
  else if (N == 2)
    *reinterpret_cast<float2*>(p) = make_float2(v[0], v[N > 1 ? 1 : 0]);
  else
    *p = v[0];
}

template <int N>
__device__ __forceinline__ void reduce_into(float* p, const float (&v)[N]) {
  if (N == 4)
    red_add_v4(p, make_float4(v[0], v[N > 1 ? 1 : 0], v[N > 2 ? 2 : 0], v[N > 3 ? 3 : 0]));
  else if (N == 2)
    asm volatile("red.global.add.v2.f32 [%0], {%1,%2};" ::"l"(p), "f"(v[0]), "f"(v[N > 1 ? 1 : 0]) : "memory");
  else
    asm volatile("red.global.add.f32 [%0], %1;" ::"l"(p), "f"(v[0]) : "memory");
}

template <int N>
__device__ __forceinline__ void load_l2(float (&d)[N], const float* p) {   // __ldcg: what other SMs wrote
  if (N == 4) {
    const float4 v = __ldcg(reinterpret_cast<const float4*>(p));
    d[0] = v.x, d[N > 1 ? 1 : 0] = v.y, d[N > 2 ? 2 : 0] = v.z, d[N > 3 ? 3 : 0] = v.w;
  } else if (N == 2) {
    const float2 v = __ldcg(reinterpret_cast<const float2*>(p));
    d[0] = v.x, d[N > 1 ? 1 : 0] = v.y;
  } else {
    d[0] = __ldcg(p);
  }
}

// Sums of the groups in every lane: partner distances 16, 8, .. down to W, the same pairing as combine_groups.
template <int VEC, int W>
__device__ __forceinline__ void all_reduce_groups(float (&a)[VEC]) {
#pragma unroll
  for (int d = 16; d >= W; d >>= 1)
#pragma unroll
    for (int x = 0; x < VEC; ++x) a[x] += __shfl_xor_sync(0xffffffffu, a[x], d);
}

// The groups' partial sums of one row fragment, combined and split over the lanes (group_split says who holds what).
// The groups split the work: each exchange hands the partner the half of the values it will own and keeps the
// other half, so four values over four groups take 3 shuffles instead of 8, and every lane writes (W = 8, VEC =
// 4: 32 lanes one float each, one 128-byte line).  When one value is left and groups remain, the rest of the
// exchange is a plain sum and one group writes.  Every kept value is own + partner in the pairing of
// all_reduce_groups, so the bits are the same.
template <int VEC, int W>
struct group_split {
  static constexpr int G = 32 / W;
  static constexpr int HALVES = VEC == 4 ? 2 : (VEC == 2 ? 1 : 0);   // halvings a fragment allows
  static constexpr int LEVELS = G == 1 ? 0 : G == 2 ? 1 : G == 4 ? 2 : G == 8 ? 3 : G == 16 ? 4 : 5;
  static constexpr int SPLITS = HALVES < LEVELS ? HALVES : LEVELS;
  static constexpr int KEEP = VEC >> SPLITS;                          // values a lane is left with
  static constexpr int REST = ((32 >> SPLITS) - 1) & ~(W - 1);        // lanes with these bits clear write
  // first column (inside the group's fragment) of the values a lane is left with
  static __device__ __forceinline__ int column(int lane) {
    int c = (lane & (W - 1)) * VEC;
    if (SPLITS >= 1) c += (lane & 16) ? VEC / 2 : 0;
    if (SPLITS >= 2) c += (lane & 8) ? VEC / 4 : 0;
    return c;
  }
  static __device__ __forceinline__ bool writes(int lane) { return REST == 0 || (lane & REST) == 0; }
};

template <int VEC, int W>
__device__ __forceinline__ void combine_groups(const float (&a)[VEC], float (&out)[group_split<VEC, W>::KEEP], int lane) {
  using S = group_split<VEC, W>;
  float k[VEC];
#pragma unroll
  for (int x = 0; x < VEC; ++x) k[x] = a[x];
#pragma unroll
  for (int s = 0; s < S::SPLITS; ++s) {
    const int d = 16 >> s, n = VEC >> (s + 1);
    const bool up = (lane & d) != 0;
#pragma unroll
    for (int x = 0; x < VEC / 2; ++x)
      if (x < n) {
        const float send = up ? k[x] : k[x + n];
        const float keep = up ? k[x + n] : k[x];
        k[x] = keep + __shfl_xor_sync(0xffffffffu, send, d);
      }
  }
#pragma unroll
  for (int s = S::SPLITS; s < S::LEVELS; ++s)
#pragma unroll
    for (int x = 0; x < S::KEEP; ++x) k[x] += __shfl_xor_sync(0xffffffffu, k[x], 16 >> s);
#pragma unroll
  for (int x = 0; x < S::KEEP; ++x) out[x] = k[x];
}

// log2 of a power of two
__host__ __device__ constexpr int ilog2(int n) { return n <= 1 ? 0 : 1 + ilog2(n / 2); }

// Sums p[0..U-1] over the W lanes of a group.  While values remain to be split, each exchange hands the partner
// half of them; afterwards lane l holds in the return value the total of entry `which(l)`.
template <int U, int W>
__device__ __forceinline__ float reduce_transposed(float (&p)[U], int lane) {
  int n = U, d = 1;
#pragma unroll
  for (int s = 0; s < ilog2(U); ++s) {
    const bool up = (lane & d) != 0;
    n >>= 1;
#pragma unroll
    for (int i = 0; i < U / 2; ++i)
      if (i < n) {
        const float send = up ? p[i] : p[i + n];
        const float keep = up ? p[i + n] : p[i];
        p[i] = keep + __shfl_xor_sync(0xffffffffu, send, d);
      }
    d <<= 1;
  }
  float total = p[0];
#pragma unroll
  for (int s = ilog2(U); s < ilog2(W); ++s) {
    total += __shfl_xor_sync(0xffffffffu, total, d);
    d <<= 1;
  }
  return total;
}

template <int U>
__device__ __forceinline__ int reduced_entry(int l) {   // the entry whose total lane l < U holds: l with its bits reversed
  int w = 0;
#pragma unroll
  for (int s = 0; s < ilog2(U); ++s) w |= ((l >> s) & 1) << (ilog2(U) - 1 - s);
  return w;
}

}  // namespace hpspmm

// Instances of the CSR product kernel for even widths that are not multiples of 4 (8-byte gathers).
#include "spmm_warp.cuh"
using namespace hpspmm;

int hpspmm_spmm_launch_v2(hpspmm_ctx* ctx, const hpspmm_spmm_args& a, const hpspmm_spmm_shape& sh, bool shared,
                          cudaStream_t s) {
#define GO(W, R, U, MINB) return launch_spmm_shape<2, W, R, U, 0, MINB, true>(ctx, a, shared, s)
  if (sh.lat) {
    if (sh.W == 16) GO(16, 1, 16, 8);
    if (sh.W == 32 && sh.R == 1) GO(32, 1, 16, 8);
    if (sh.W == 32 && sh.R == 2) GO(32, 2, 16, 8);
    if (sh.W == 32 && sh.R == 3) GO(32, 3, 8, 8);
    if (sh.W == 32) GO(32, 4, 8, 8);
  }
  if (sh.W == 2) GO(2, 1, 2, 16);
  if (sh.W == 4) GO(4, 1, 4, 16);
  if (sh.W == 8) GO(8, 1, 8, 16);
  if (sh.W == 16 && sh.R == 3) GO(16, 3, 4, 18);
  if (sh.W == 16) GO(16, 1, 8, 18);
  if (sh.R == 1) GO(32, 1, 8, 18);
  if (sh.R == 2) GO(32, 2, 4, 18);
  if (sh.R == 3) GO(32, 3, 2, 18);
  GO(32, 4, 2, 18);
#undef GO
}

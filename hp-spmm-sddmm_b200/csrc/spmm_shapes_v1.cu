// Instances of the CSR product kernel for odd widths (4-byte gathers).
#include "spmm_warp.cuh"
using namespace hpspmm;

int hpspmm_spmm_launch_v1(hpspmm_ctx* ctx, const hpspmm_spmm_args& a, const hpspmm_spmm_shape& sh, bool shared,
                          cudaStream_t s) {
#define GO(W, R, U, MINB) return launch_spmm_shape<1, W, R, U, 0, MINB, true>(ctx, a, shared, s)
  if (sh.lat) {
    if (sh.W == 16) GO(16, 1, 16, 8);
    if (sh.W == 32 && sh.R == 1) GO(32, 1, 32, 8);
    if (sh.W == 32 && sh.R == 2) GO(32, 2, 16, 8);
    if (sh.W == 32 && sh.R == 3) GO(32, 3, 8, 8);
    if (sh.W == 32 && sh.R == 4) GO(32, 4, 8, 8);
  }
  if (sh.W == 1) GO(1, 1, 1, 16);
  if (sh.W == 4) GO(4, 1, 4, 16);
  if (sh.W == 8) GO(8, 1, 8, 16);
  if (sh.W == 16 && sh.R == 3) GO(16, 3, 4, 18);
  if (sh.W == 16) GO(16, 1, 8, 18);
  if (sh.R == 1) GO(32, 1, 8, 18);
  if (sh.R == 2) GO(32, 2, 8, 18);
  if (sh.R == 3) GO(32, 3, 4, 18);
  if (sh.R == 4) GO(32, 4, 4, 18);
  if (sh.R == 5) GO(32, 5, 2, 18);
  if (sh.R == 6) GO(32, 6, 2, 18);
  if (sh.R == 7) GO(32, 7, 2, 18);
  GO(32, 8, 2, 18);
#undef GO
}

// Instances of the CSR product kernel for widths that are multiples of 4 (16-byte gathers).
#include "spmm_warp.cuh"
using namespace hpspmm;

int hpspmm_spmm_launch_v4(hpspmm_ctx* ctx, const hpspmm_spmm_args& a, const hpspmm_spmm_shape& sh, bool shared,
                          cudaStream_t s) {
#define GO(W, R, U, KS, MINB, H) return launch_spmm_shape<4, W, R, U, KS, MINB, H>(ctx, a, shared, s)
  if (sh.lat) {
    if (sh.W == 8) GO(8, 1, 8, 0, 12, true);
    if (sh.W == 16) GO(16, 1, 16, 0, 8, true);
    if (sh.W == 32 && sh.R == 1) GO(32, 1, 16, 0, 8, true);
    if (sh.W == 32 && sh.R == 2) GO(32, 2, 8, 0, 8, true);
    if (sh.W == 32 && sh.R == 3) GO(32, 3, 4, 0, 8, true);
    if (sh.W == 32) GO(32, 4, 4, 0, 8, true);
  }
  if (sh.mid) {
    if (sh.R == 1) GO(32, 1, 8, 0, 12, true);
    GO(32, 2, 4, 0, 12, true);
  }
  if (a.K == 32 && sh.W == 8) { if (sh.hint) GO(8, 1, 4, 32, 18, true); else GO(8, 1, 4, 32, 18, false); }
  if (a.K == 64 && sh.W == 16) { if (sh.hint) GO(16, 1, 4, 64, 18, true); else GO(16, 1, 4, 64, 18, false); }
  if (a.K == 128 && sh.W == 32 && sh.R == 1) { if (sh.hint) GO(32, 1, 4, 128, 18, true); else GO(32, 1, 4, 128, 18, false); }
  if (sh.W == 2) GO(2, 1, 2, 0, 16, true);
  if (sh.W == 4) GO(4, 1, 4, 0, 16, true);
  if (sh.W == 8 && sh.R == 3) GO(8, 3, 2, 0, 16, true);
  if (sh.W == 8) GO(8, 1, 4, 0, 16, true);
  if (sh.W == 16 && sh.R == 3) GO(16, 3, 2, 0, 16, true);
  if (sh.W == 16) GO(16, 1, 4, 0, 18, true);
  if (sh.R == 1) GO(32, 1, 4, 0, 18, true);
  if (sh.R == 2) GO(32, 2, 2, 0, 18, true);
  if (sh.R == 3) GO(32, 3, 2, 0, 12, true);
  GO(32, 4, 1, 0, 12, true);
#undef GO
}

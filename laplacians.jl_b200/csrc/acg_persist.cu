// The one-vector kernels, in a module of their own.  Their time depends on where
// their code lies: with all kernels in one module, k_pcg became 2 to 12 % slower
// with a change to kernels that it never calls (us per iteration: 32 x 32 grid
// 13.0 and 13.5, 200 x 200 grid 49.9 and 52.8, a geometric graph of 1,319
// vertices in mixed precision 16.2 and 18.6).  Here their place does not move
// with other kernels' code, and the times are the lower ones (13.0, 50.1, 16.0).
#include "acg_persist.cuh"

namespace acg {
ACG_PERSIST_KERNELS(template)
}  // namespace acg

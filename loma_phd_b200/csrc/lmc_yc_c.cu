// y kernels for chunks of 9 rows, 16 modes per block (see lmc_ychunk.cuh).
#include "lmc_ychunk.cuh"

namespace lmc {
template struct YC<9, 16>;
}  // namespace lmc

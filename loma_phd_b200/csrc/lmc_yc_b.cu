// y kernels for chunks of 9 rows, 8 modes per block (see lmc_ychunk.cuh).
#include "lmc_ychunk.cuh"

namespace lmc {
template struct YC<9, 8>;
}  // namespace lmc

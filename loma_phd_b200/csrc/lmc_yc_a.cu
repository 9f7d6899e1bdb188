// y kernels for chunks of 5 rows, 8 modes per block (see lmc_ychunk.cuh).
#include "lmc_ychunk.cuh"

namespace lmc {
template struct YC<5, 8>;
}  // namespace lmc

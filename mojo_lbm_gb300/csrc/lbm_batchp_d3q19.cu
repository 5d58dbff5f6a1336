// The 16 double-buffer batched-step variants of the D3Q19 lattice with two cells per thread.
#include "lbm_batch.cuh"

namespace lbm {
BatchLaunch get_batch_pair_step_d3q19(int f16c, int coll, int les) {
    static const BatchLaunch t[16] = LBM_DB_TABLE(launch_step_batch_pair, D3Q19);
    return t[db_index(f16c, coll, les)];
}
}  // namespace lbm

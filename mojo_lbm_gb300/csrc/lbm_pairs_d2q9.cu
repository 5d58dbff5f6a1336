// The 16 esoteric-pull cell-pair fused-step variants of the D2Q9 lattice in the fast arithmetic
// (lbm_pair.cuh).
#include "lbm_pair.cuh"

namespace lbm {
StepLaunch get_pair_eso_step_d2q9(int f16c, int coll, int les) {
    static const StepLaunch fast[16] = LBM_ESO_TABLE(launch_step_pair_fast, D2Q9);
    return fast[db_index(f16c, coll, les)];
}
}  // namespace lbm

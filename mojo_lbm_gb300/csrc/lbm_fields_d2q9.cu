// The initial-state and output kernels of the D2Q9 lattice (lbm_fields.cuh).
#include "lbm_fields.cuh"

namespace lbm {
cudaError_t launch_init_d2q9(const InitArgs& a, bool f16, cudaStream_t s) { return launch_init<D2Q9>(a, f16, s); }
cudaError_t launch_rho_u_d2q9(const RhoUArgs& a, bool f16, bool eso, bool qcrit, cudaStream_t s) {
    return launch_rho_u<D2Q9>(a, f16, eso, qcrit, s);
}
}  // namespace lbm

// kernels_diag_f64.cu -- diagnostics of FP64 fields (compiled with --fmad=false,
// as kernels_f64.cu: the director and the plaquette signs are the reference's).
#include "diag_launch.cuh"

LBMAN_DEFINE_DIAG(f64, double)

namespace lbman {
cudaError_t launch_fold(const double* partials, int G, int nq, int nmax, double* out, cudaStream_t st) {
    fold_partials_kernel<<<1, 1024, 0, st>>>(partials, G, nq, nmax, out);
    return cudaGetLastError();
}
}  // namespace lbman

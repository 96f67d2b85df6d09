// k_eri_s.cu — the three-centre integral kernels (eri_thread.cuh) for aux shells of l = 0; one file per l so
// that the straight-line recursions compile in parallel.
#include "eri_thread.cuh"

namespace rijk {
namespace eri {
template cudaError_t launch_lc<0>(int lab, const EriLaunch& P, size_t smem, cudaStream_t s);
}  // namespace eri
}  // namespace rijk

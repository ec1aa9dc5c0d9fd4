// Instantiations of the batched Lanczos kernel.
#include "ed_batch_kernel.cuh"

namespace ed {
template ed_status launch_batch<512, 2>(const ed_batch_s*, int, int, int, double, int, uint64_t, const double* const*,
                                        int, const BatchOut&, const BatchWork&, cudaStream_t);
template int clusters_for<512, 2>();
template ed_status launch_batch<1024, 2>(const ed_batch_s*, int, int, int, double, int, uint64_t, const double* const*,
                                        int, const BatchOut&, const BatchWork&, cudaStream_t);
template int clusters_for<1024, 2>();
}  // namespace ed

// Instantiations of the batched Lanczos kernel.
#include "ed_batch_kernel.cuh"

namespace ed {
template ed_status launch_batch<288, 1>(const ed_batch_s*, int, int, int, double, int, uint64_t, const double* const*,
                                        int, const BatchOut&, const BatchWork&, cudaStream_t);
template ed_status launch_batch<544, 1>(const ed_batch_s*, int, int, int, double, int, uint64_t, const double* const*,
                                        int, const BatchOut&, const BatchWork&, cudaStream_t);
template ed_status launch_batch<800, 1>(const ed_batch_s*, int, int, int, double, int, uint64_t, const double* const*,
                                        int, const BatchOut&, const BatchWork&, cudaStream_t);
}  // namespace ed

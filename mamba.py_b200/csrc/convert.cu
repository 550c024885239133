// Small element-wise jobs of a layer, many in one launch: parameters to the types and layouts the kernels take before a
// forward, gradients back to the parameters' types after a backward.  A job is a (rows, cols) matrix; each is a few
// thousand to a few hundred thousand elements, so what counts is the number of launches, not the bandwidth: one launch of
// 3 us replaces the 6 to 10 that separate casts, exponentials and products took.
#include "convert.cuh"

namespace mb200 {
namespace {

constexpr int kMaxJobs = MB200_CONVERT_MAX_JOBS;

__global__ void __launch_bounds__(kConvertThreads) convert_kernel(const __grid_constant__ Jobs<kMaxJobs> jobs) {
  convert_block(jobs, int(blockIdx.x));
}

}  // namespace
}  // namespace mb200

using namespace mb200;

extern "C" int mb200_convert(const mb200_convert_job* jobs, int n, void* stream) {
  Jobs<kMaxJobs> all;
  int64_t blocks = 0;
  const int rc = collect_jobs(jobs, n, all, blocks);
  if (rc != MB200_OK || all.n == 0) return rc;
  convert_kernel<<<unsigned(blocks), kConvertThreads, 0, static_cast<cudaStream_t>(stream)>>>(all);
  return check_launch();
}

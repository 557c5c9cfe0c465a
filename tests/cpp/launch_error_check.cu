// launch_kernel() over a fake runtime: prints whether a failed launch returns its error, the last error left behind by it,
// the result of a good launch, and how many of the two launches asked to start early.
#include <cstdio>

#include "../../godunov_mhd_ct_gb300/csrc/launch.cuh"

extern cudaError_t fake_launch_result, fake_last_error;
extern int         fake_early_launches;

static void
kernel(int)
{
}

int
main()
{
  fake_launch_result = cudaErrorStreamCaptureImplicit;
  const cudaError_t bad = gmhd::launch_kernel(kernel, 1u, 32, (size_t)0, (cudaStream_t)0, true, 1), left = fake_last_error;
  fake_launch_result = fake_last_error = cudaSuccess;
  const cudaError_t good = gmhd::launch_kernel(kernel, 1u, 32, (size_t)0, (cudaStream_t)0, false, 1);
  std::printf("%d %d %d %d\n", bad == cudaErrorStreamCaptureImplicit, (int)left, (int)good, fake_early_launches);
  return 0;
}

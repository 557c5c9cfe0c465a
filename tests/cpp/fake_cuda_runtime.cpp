// Stands in for the CUDA runtime in launch_error_check: the two calls that launch_kernel() makes, and what the compiler's
// startup code refers to.
#include <cuda_runtime_api.h>

cudaError_t fake_launch_result = cudaSuccess, fake_last_error = cudaSuccess;
int         fake_early_launches = 0;

extern "C" cudaError_t
cudaLaunchKernelExC(const cudaLaunchConfig_t * cfg, const void *, void **)
{
  fake_early_launches += (int)cfg->numAttrs;
  if (fake_launch_result != cudaSuccess)
    fake_last_error = fake_launch_result;
  return fake_launch_result;
}
extern "C" cudaError_t
cudaGetLastError()
{
  const cudaError_t e = fake_last_error;
  fake_last_error = cudaSuccess;
  return e;
}
extern "C" void **
__cudaRegisterFatBinary(void *)
{
  return nullptr;
}
extern "C" void
__cudaRegisterFatBinaryEnd(void **)
{
}
extern "C" void
__cudaUnregisterFatBinary(void **)
{
}
extern "C" char
__cudaInitModule(void **)
{
  return 0;
}

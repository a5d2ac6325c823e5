// A launch that CUDA refuses (more threads than a block can have, or no device
// at all) throws at once, whatever the calls after it do with the last error.
#include <cstdio>

#include "engine.h"

__global__ void k_nothing(int *) {}

int main()
{
  try
  {
    qm::launch_kernel(k_nothing, 1, 4096, 0, nullptr, 0, (int *)nullptr);
  }
  catch (const qm::CudaError &e)
  {
    std::printf("%s\n", e.msg.c_str());
    return 3;
  }
  return 0;
}

// A launch of one thread that lets its dependents start at once and then waits `ms` milliseconds: the longest a launch can keep others that
// are set up under its end.
#include <cuda_runtime.h>
#include <stdint.h>

__global__ void early_trigger_kernel(uint64_t ns) {
  uint64_t t0, t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  asm volatile("griddepcontrol.wait;\n\tgriddepcontrol.launch_dependents;" ::: "memory");
  do {
    __nanosleep(100000);
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  } while (t - t0 < ns);
}

extern "C" int early_trigger(int ms, void* stream) {
  if (ms < 0 || ms > 4000) return -1;
  early_trigger_kernel<<<1, 1, 0, static_cast<cudaStream_t>(stream)>>>((uint64_t)ms * 1000000ull);
  return (int)cudaGetLastError();
}

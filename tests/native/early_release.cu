// A caller's kernel that lets the next kernel of its stream start at once and then runs on for `ns`
// nanoseconds (at most `rounds` sleeps of about a microsecond); built by tests/test_gpu_early_release.py.
#include <cuda_runtime.h>

static __global__ void early_release_kernel(unsigned long long ns, unsigned rounds) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    unsigned long long start, now;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(start));
    for (unsigned i = 0; i < rounds; ++i) {
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        if (now - start >= ns) return;
        __nanosleep(1000);
    }
}

extern "C" int early_release(unsigned long long ns, unsigned rounds, void* stream) {
    early_release_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(ns, rounds);
    return int(cudaGetLastError());
}

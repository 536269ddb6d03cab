// wp_shape.cu -- launch shapes of kernels with dynamic shared memory, kept per
// device: how many CTAs share an SM, and the function attribute that allows the
// shared memory.  A small classify call spent some 2 us of host time per launch
// on asking again.
#include <cuda_runtime.h>

#include <map>
#include <mutex>
#include <tuple>

// CTAs of `threads` threads and `smem` bytes of dynamic shared memory per SM of
// the current device (*per_sm, 0 if none fits) and its SMs (*sms); the kernel may
// be launched with that much shared memory afterwards.  Safe from several
// threads: the attribute only ever grows.
cudaError_t wp_launch_shape(const void* kernel, int threads, size_t smem, int* per_sm, int* sms) {
    struct Shape {
        int per_sm, sms;
    };
    static std::mutex mu;
    static std::map<std::tuple<const void*, int, int, size_t>, Shape> shapes;
    static std::map<std::pair<const void*, int>, size_t> allowed;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(mu);
    const auto key = std::make_tuple(kernel, dev, threads, smem);
    const auto it = shapes.find(key);
    if (it != shapes.end()) {
        *per_sm = it->second.per_sm;
        *sms = it->second.sms;
        return cudaSuccess;
    }
    size_t& have = allowed[{kernel, dev}];
    if (smem > have) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        have = smem;
    }
    Shape s = {0, 0};
    e = cudaDeviceGetAttribute(&s.sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&s.per_sm, kernel, threads, smem);
    if (e != cudaSuccess) return e;
    shapes[key] = s;
    *per_sm = s.per_sm;
    *sms = s.sms;
    return cudaSuccess;
}

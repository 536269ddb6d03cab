// wp_shape.cu -- launch shapes of kernels with dynamic shared memory, kept per
// device: how many CTAs share an SM, and the function attribute that allows the
// shared memory.  A small classify call spent some 2 us of host time per launch
// on asking again.
#include <cuda_runtime.h>

#include <map>
#include <mutex>
#include <tuple>

namespace {
struct Shape {
    int per_sm, sms;
};
constexpr size_t MOST = 4096;  // shapes kept
std::mutex mu;
std::map<std::tuple<const void*, int, int, size_t>, Shape> shapes;
}  // namespace

// CTAs of `threads` threads and `smem` bytes of dynamic shared memory per SM of
// the current device (*per_sm, 0 if none fits) and its SMs (*sms); the kernel may
// be launched with that much shared memory afterwards.  Safe from several
// threads: the attribute only ever grows.
cudaError_t wp_launch_shape(const void* kernel, int threads, size_t smem, int* per_sm, int* sms) {
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
    cudaFuncAttributes attr;
    e = cudaFuncGetAttributes(&attr, kernel);
    if (e == cudaSuccess && (size_t)attr.maxDynamicSharedSizeBytes < smem)
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    Shape s = {0, 0};
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&s.sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&s.per_sm, kernel, threads, smem);
    if (e != cudaSuccess) return e;
    try {
        if (shapes.size() >= MOST) shapes.clear();
        shapes[key] = s;
    } catch (...) {
        // not kept: asked again next time
    }
    *per_sm = s.per_sm;
    *sms = s.sms;
    return cudaSuccess;
}

// Forgets the shapes (a new context: the device may have been reset since, and
// its function attributes with it).
void wp_launch_shape_forget() {
    std::lock_guard<std::mutex> lk(mu);
    shapes.clear();
}

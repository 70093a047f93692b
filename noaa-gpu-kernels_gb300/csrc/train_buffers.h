// Device buffers of the training launches (warm.cu), host side only, so that their
// sizes can be checked without a device.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>

namespace tr {

constexpr int kTrainRows = 64;   // samples per tile
constexpr int kPartLd = 4804;    // row of the partial gradients, 16-byte aligned

// AdamW constants of a step.
struct AdamStep {
    float lr, c1, c2;
};

// Steps per launch: their samples' losses are kept and summed afterwards (64 doubles
// in order take as long as a tile's products).
inline int train_steps_kept(long long steps_per_epoch, int tiles)
{
    return (int)std::min<long long>(steps_per_epoch, std::max(1, (1 << 16) / tiles));
}

// One buffer with a count of its own: a call may need more of one buffer and less of
// another than the call before it, so no buffer's size stands for another's.
template <typename T>
struct TrainBuf {
    T* p = nullptr;
    size_t n = 0;   // elements allocated
    cudaError_t reserve(size_t need)
    {
        if (need <= n) return cudaSuccess;
        release();
        const cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&p), need * sizeof(T));
        if (e == cudaSuccess) n = need;
        else p = nullptr;
        return e;
    }
    void release()
    {
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
    }
    TrainBuf() = default;
    TrainBuf(const TrainBuf&) = delete;
    TrainBuf& operator=(const TrainBuf&) = delete;
    ~TrainBuf() { release(); }
};

// What `steps` steps of `tiles` tiles write: a row of partial gradients a tile (used
// again by every step), a loss a tile and one a step, every sample's (err^2)/2, and
// the steps' constants.
struct TrainBuffers {
    TrainBuf<float> part, err;
    TrainBuf<double> loss;
    TrainBuf<AdamStep> step;
    cudaError_t reserve(int tiles, int steps)
    {
        const size_t t = (size_t)tiles, s = (size_t)steps;
        cudaError_t e = part.reserve(t * kPartLd);
        if (e == cudaSuccess) e = err.reserve(s * t * kTrainRows);
        if (e == cudaSuccess) e = loss.reserve(s * t + s);
        if (e == cudaSuccess) e = step.reserve(s);
        return e;
    }
};

}  // namespace tr

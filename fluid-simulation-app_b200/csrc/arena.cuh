// arena.cuh — many device buffers as one allocation.
//
// An adjoint's tape is over a thousand buffers: the first backward of the
// 64k-particle workload spent 170 ms in cudaMalloc, and 2 ms with the
// buffers asked for first and placed in one block. (The simulations' 40
// buffers stay on their own: small ones come out of the driver's pools,
// and one large block measured slower to create.)
#pragma once

#include <cuda_runtime.h>

#include <utility>
#include <vector>

namespace fcu {

class Arena {
    std::vector<std::pair<void **, size_t>> wanted_;
    std::vector<void *> blocks_;

public:
    // Asks for `count` elements; *p is set by the next commit().
    template <class T>
    void want(T **p, size_t count) {
        const size_t bytes = (count ? count : 1) * sizeof(T);
        wanted_.emplace_back(reinterpret_cast<void **>(p), (bytes + 255) & ~(size_t)255);
    }
    // Allocates everything asked for since the last commit, each buffer
    // 256-byte aligned.
    cudaError_t commit() {
        size_t total = 0;
        for (const auto &w : wanted_) total += w.second;
        void *block = nullptr;
        const cudaError_t e = cudaMalloc(&block, total ? total : 256);
        if (e == cudaSuccess) {
            blocks_.push_back(block);
            char *at = static_cast<char *>(block);
            for (const auto &w : wanted_) {
                *w.first = at;
                at += w.second;
            }
        }
        wanted_.clear();
        return e;
    }
    // Frees every block (the device current).
    void release() {
        for (void *b : blocks_) cudaFree(b);
        blocks_.clear();
    }
};

}  // namespace fcu

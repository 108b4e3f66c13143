// io_scratch.h — device scratch of the mesh-file calls (decoders, weld, orientation).
//
// A call takes a dozen to two dozen arrays. They are carved from one block kept per device;
// what does not fit is allocated for the call, and a call that outgrew the block leaves it
// large enough for the next of its size (up to kIoKept; gbsdf_release_workspace gives it
// back). Allocating and freeing every array on each call took 0.7 of the 1.1 ms of decoding a
// 9 MB binary STL. One call at a time holds the block; calls that find it taken allocate.
#pragma once

#include <algorithm>
#include <vector>

#include <cuda_runtime.h>

namespace gbsdf {

constexpr size_t kIoKept = size_t(512) << 20;  // most bytes kept per device

// (defined in k_io.cu)
bool io_block_take(int device, void** base, size_t* bytes);
void io_block_give(int device, size_t want);  // grown to `want` bytes if it held fewer
void release_io_workspace(int device);

class IoScratch {
public:
    explicit IoScratch(int device) : device_(device), held_(io_block_take(device, &base_, &bytes_)) {}
    ~IoScratch() {
        for (void* p : ptrs_) cudaFree(p);
        if (held_) io_block_give(device_, need_ <= kIoKept ? need_ : 0);
    }
    IoScratch(const IoScratch&) = delete;
    IoScratch& operator=(const IoScratch&) = delete;
    template <class T>
    T* get(size_t count, cudaError_t& err) {
        if (err != cudaSuccess) return nullptr;
        const size_t b = (std::max<size_t>(count, 1) * sizeof(T) + 255) & ~size_t(255);
        need_ += b;
        if (held_ && used_ + b <= bytes_) {
            void* p = static_cast<char*>(base_) + used_;
            used_ += b;
            return static_cast<T*>(p);
        }
        void* p = nullptr;
        err = cudaMalloc(&p, b);
        if (err != cudaSuccess) return nullptr;
        ptrs_.push_back(p);
        return static_cast<T*>(p);
    }

private:
    int device_;
    void* base_ = nullptr;
    size_t bytes_ = 0, used_ = 0, need_ = 0;
    bool held_;
    std::vector<void*> ptrs_;
};

}  // namespace gbsdf

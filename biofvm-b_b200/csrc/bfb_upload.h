// bfb_upload.h -- host-to-device copies whose sources outlive them (host).
//
// cudaMemcpyAsync may read a pageable source after it has returned, so a table
// made in a local vector has to live until the stream has been waited for. An
// Uploads object takes such buffers over, and its wait (or its end, on an error
// return) waits for the stream before it frees them. One wait covers all tables
// of a call.
#pragma once
#include <cuda_runtime_api.h>

#include <memory>
#include <utility>
#include <vector>

namespace bfb {

class Uploads {
  public:
    explicit Uploads(cudaStream_t s) : s_(s) {}
    Uploads(const Uploads &) = delete;
    Uploads &operator=(const Uploads &) = delete;
    ~Uploads() { wait(); }

    // a buffer handed over with std::move
    template <typename V>
    cudaError_t copy(void *dst, std::vector<V> &&src) {
        const std::vector<V> &v = keep(std::move(src));
        return copy(dst, v.data(), v.size() * sizeof(V));
    }
    // a buffer of the caller's, which has to outlive this object
    cudaError_t copy(void *dst, const void *src, size_t bytes) {
        pending_ = true;
        return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s_);
    }
    // packed rows of row_bytes into rows dst_pitch bytes apart; a buffer handed over
    template <typename V>
    cudaError_t copy_rows(void *dst, size_t dst_pitch, std::vector<V> &&src, size_t row_bytes, size_t rows) {
        const std::vector<V> &v = keep(std::move(src));
        pending_ = true;
        return cudaMemcpy2DAsync(dst, dst_pitch, v.data(), row_bytes, row_bytes, rows, cudaMemcpyHostToDevice, s_);
    }
    // Waits for the stream, then lets the buffers go.
    cudaError_t wait() {
        const cudaError_t e = pending_ ? cudaStreamSynchronize(s_) : cudaSuccess;
        pending_ = false;
        kept_.clear();
        return e;
    }

  private:
    template <typename V>
    const std::vector<V> &keep(std::vector<V> &&src) {
        auto p = std::make_shared<std::vector<V>>(std::move(src));
        kept_.push_back(p);
        return *p;
    }
    cudaStream_t s_;
    bool pending_ = false;
    std::vector<std::shared_ptr<void>> kept_;
};

}  // namespace bfb

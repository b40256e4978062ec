// csrc/bfb_upload.h against a CUDA runtime that reads no source before the
// stream is waited for (the latest that cudaMemcpyAsync allows): every byte has
// to arrive although the callers' vectors are gone by then. Prints "ok".
#include "bfb_upload.h"

#include <cstdio>
#include <cstring>
#include <functional>

static std::vector<std::function<void()>> queued;
static int waits = 0;

extern "C" cudaError_t CUDARTAPI cudaMemcpyAsync(void *dst, const void *src, size_t n, cudaMemcpyKind, cudaStream_t) {
    queued.push_back([=] { std::memcpy(dst, src, n); });
    return cudaSuccess;
}
extern "C" cudaError_t CUDARTAPI cudaMemcpy2DAsync(void *dst, size_t dp, const void *src, size_t sp, size_t w, size_t h,
                                                   cudaMemcpyKind, cudaStream_t) {
    queued.push_back([=] {
        for (size_t r = 0; r < h; ++r) std::memcpy((char *)dst + r * dp, (const char *)src + r * sp, w);
    });
    return cudaSuccess;
}
extern "C" cudaError_t CUDARTAPI cudaStreamSynchronize(cudaStream_t) {
    ++waits;
    for (auto &q : queued) q();
    queued.clear();
    return cudaSuccess;
}

// As the library's callers: tables made in local vectors, an early return in between.
static bool stage(int *a, double *b, bool fail_early) {
    bfb::Uploads up(nullptr);
    {
        std::vector<int> v(1000);
        for (int q = 0; q < 1000; ++q) v[q] = 3 * q;
        if (up.copy(a, std::move(v)) != cudaSuccess) return false;
    }
    {
        std::vector<double> v(12);
        for (int q = 0; q < 12; ++q) v[q] = q + 0.5;
        if (up.copy_rows(b, 4 * sizeof(double), std::move(v), 3 * sizeof(double), 4) != cudaSuccess) return false;
    }
    std::vector<int> other(1000, -1);  // takes the freed memory if the first vector was let go
    if (fail_early) return other[0] == -1;
    return up.wait() == cudaSuccess && other[0] == -1;
}

int main() {
    for (bool fail_early : {false, true}) {
        std::vector<int> a(1000, 0);
        std::vector<double> b(16, -7.0);
        waits = 0;
        if (!stage(a.data(), b.data(), fail_early) || waits != 1 || !queued.empty()) return std::puts("wait"), 1;
        for (int q = 0; q < 1000; ++q)
            if (a[q] != 3 * q) return std::puts("lost"), 1;
        for (int r = 0; r < 4; ++r)
            for (int c = 0; c < 4; ++c)
                if (b[4 * r + c] != (c < 3 ? 3 * r + c + 0.5 : -7.0)) return std::puts("rows"), 1;
    }
    {
        bfb::Uploads none(nullptr);  // nothing copied: nothing to wait for
        waits = 0;
    }
    if (waits) return std::puts("idle"), 1;
    std::puts("ok");
    return 0;
}

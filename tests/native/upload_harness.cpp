// Test harness: DBuf (internal.hpp) over a CUDA runtime that holds every
// asynchronous copy back until its stream is waited for, as a copy from
// pageable host memory may be; compiled by tests/test_cpu_uploads.py.
#include <cstdlib>
#include <cstring>
#include <functional>

#include "internal.hpp"

namespace {
std::vector<std::pair<cudaStream_t, std::function<void()>>> pending;
}

extern "C" {

cudaError_t cudaMalloc(void **p, size_t n) {
    *p = std::calloc(1, n);
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    std::free(p);
    return cudaSuccess;
}
const char *cudaGetErrorString(cudaError_t) { return ""; }
cudaError_t cudaMemcpyAsync(void *to, const void *from, size_t n, cudaMemcpyKind, cudaStream_t s) {
    pending.push_back({s, [=] { std::memcpy(to, from, n); }});
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    for (auto &c : pending)
        if (c.first == s) c.second();
    std::erase_if(pending, [&](auto &c) { return c.first == s; });
    return cudaSuccess;
}

// upload_vec of a vector that holds 0 .. n - 1 during the call and -1 from
// then on (its memory is kept, so that a late copy is seen and not a fault).
// Returns the values that arrived; -2 when a copy is still pending.
int uploaded(int n, int empty_first) {
    axgb::DBuf<int> d;
    std::vector<int> v(n);
    for (int k = 0; k < n; ++k) v[k] = k;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(1);
    if (empty_first) d.upload_vec(std::vector<int>{}, s);
    d.upload_vec(v, s);
    if (!pending.empty()) return -2;
    for (int &x : v) x = -1;
    cudaStreamSynchronize(s);
    int ok = 0;
    for (int k = 0; k < n; ++k) ok += d.p[k] == k;
    return ok;
}

}

// device_memory.hpp -- device memory that a handle owns.
#pragma once

#include <cstdint>
#include <cstdio>
#include <string>
#include <utility>
#include <cuda_runtime.h>
#include "heom_b200.h"

namespace heomhost {
int set_error(int code, const std::string& msg);
}

namespace heomrt {

template <typename T>
struct DevBuf {
    T* p = nullptr;
    size_t n = 0;
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    ~DevBuf() { reset(); }
    void reset()
    {
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
    }
    int alloc(size_t count)
    {
        reset();
        if (count == 0) count = 1;
        cudaError_t e = cudaMalloc(&p, count * sizeof(T));
        if (e != cudaSuccess) {
            cudaGetLastError(); // reported here: not for the next launch's check to find
            p = nullptr;
            char buf[160];
            snprintf(buf, sizeof buf, "cudaMalloc of %zu bytes failed: %s", count * sizeof(T), cudaGetErrorString(e));
            return heomhost::set_error(HEOM_E_NOMEM, buf);
        }
        n = count;
        return 0;
    }
    // at least `count` elements; what is large enough is kept, contents and all.  After a failure the buffer is empty
    // and says so, and the next call tries again.
    int ensure(size_t count) { return p && n >= count ? 0 : alloc(count); }
    void swap(DevBuf& o)
    {
        std::swap(p, o.p);
        std::swap(n, o.n);
    }
};

// The adjoint states of a group of steps, whose gradient contributions are then one launch.  The sweep works without
// it, one launch per factor (group 0): memory that cannot be had costs speed, not the call.
template <typename T>
struct AdjointRing {
    DevBuf<T> states;
    int64_t group = 0; // steps

    // states for groups of `want` steps, `step` elements each; true when what a captured sweep holds has changed
    bool resize(int64_t want, size_t step)
    {
        const int64_t had = group;
        const T* const at = states.p;
        if (want == 0) states.reset();
        group = want;
        if (want > 0 && states.ensure((size_t)want * step) != 0) group = 0;
        return group != had || states.p != at;
    }
};

} // namespace heomrt

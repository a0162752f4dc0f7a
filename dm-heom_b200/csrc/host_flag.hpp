// host_flag.hpp -- flags that kernels set and the host reads.
#pragma once

#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <vector>
#include <cuda_runtime.h>
#include "heom_b200.h"

namespace heomhost {
int set_error(int code, const std::string& msg);
}

namespace heomrt {

// Flags that kernels set and the host reads after the stream has drained: mapped pinned memory, so that a call that
// checks one needs no copy of its own.  Page-locking takes longer than the rest of a small handle's creation, so the
// handles on a device share a page of flags, and the page stays for the handles to come: 4 KB per device until the
// process ends (a full page makes place for a new one and goes with the last of its flags).  A reset of the device
// takes its page along; the mark tells such a page, or another's memory at its address, from the live one.
struct FlagPage {
    static constexpr int kFlags = 1024, kMark = 4; // the mark lies in the first flags' place
    int* host = nullptr;
    int* dev = nullptr;
    std::vector<int> unused;
    std::mutex mu;
    FlagPage() = default;
    FlagPage(const FlagPage&) = delete;
    FlagPage& operator=(const FlagPage&) = delete;
    ~FlagPage()
    {
        if (host && live()) cudaFreeHost(host);
    }
    int alloc()
    {
        unused.reserve(kFlags); // a flag is given back without an allocation
        cudaError_t e = cudaHostAlloc(&host, kFlags * sizeof(int), cudaHostAllocMapped);
        if (e != cudaSuccess) {
            host = nullptr;
        } else if ((e = cudaHostGetDevicePointer(&dev, host, 0)) == cudaSuccess) {
            std::memcpy(host, mark(), kMark * sizeof(int));
            for (int q = kFlags - 1; q >= kMark; --q) unused.push_back(q);
            return 0;
        }
        cudaGetLastError(); // reported here: not for the next launch's check to find
        return heomhost::set_error(HEOM_E_NOMEM, std::string("mapped flags: ") + cudaGetErrorString(e));
    }
    bool live() const
    {
        cudaPointerAttributes a{};
        const bool known = cudaPointerGetAttributes(&a, host) == cudaSuccess;
        if (!known) cudaGetLastError();
        return known && a.type == cudaMemoryTypeHost && std::memcmp(host, mark(), kMark * sizeof(int)) == 0;
    }
    static const int* mark()
    {
        static const int m[kMark] = {0x48454f4d, 0x464c4147, 0x50414745, 0x2d313032};
        return m;
    }
};

struct HostFlag {
    std::shared_ptr<FlagPage> page;
    int index = -1;
    int* dev = nullptr;
    HostFlag() = default;
    HostFlag(const HostFlag&) = delete;
    HostFlag& operator=(const HostFlag&) = delete;
    ~HostFlag()
    {
        if (!page) return;
        std::lock_guard<std::mutex> lock(page->mu);
        page->unused.push_back(index);
    }
    // a flag for the kernels of the current device, whose number the caller knows
    int alloc(int device)
    {
        // never destroyed: the pages of a process that ends go with it, not by calls into a driver that is leaving too
        static std::mutex& mu = *new std::mutex;
        static std::map<int, std::shared_ptr<FlagPage>>& pages = *new std::map<int, std::shared_ptr<FlagPage>>;
        std::lock_guard<std::mutex> lock(mu);
        std::shared_ptr<FlagPage>& pg = pages[device];
        bool usable = pg && pg->live();
        if (usable) {
            std::lock_guard<std::mutex> pl(pg->mu);
            usable = !pg->unused.empty();
        }
        if (!usable) {
            std::shared_ptr<FlagPage> fresh = std::make_shared<FlagPage>();
            if (int rc = fresh->alloc()) return rc;
            pg = fresh;
        }
        std::lock_guard<std::mutex> pl(pg->mu);
        index = pg->unused.back();
        pg->unused.pop_back();
        page = pg;
        dev = pg->dev + index;
        clear();
        return 0;
    }
    void clear() { static_cast<volatile int*>(page->host)[index] = 0; }
    bool set() const { return static_cast<volatile int*>(page->host)[index] != 0; }
};

} // namespace heomrt

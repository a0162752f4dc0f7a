// Host-only check of dm-heom_b200/csrc/host_flag.hpp over a fake of the CUDA calls that it makes (compiled by
// tests/test_device_memory.py).  Prints one line per problem, then "ok" or "FAILED".
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <set>
#include <thread>
#include "host_flag.hpp"

static std::atomic<int> bad{0};
#define CHECK(x) \
    do { if (!(x)) { printf("bad line %d: %s\n", __LINE__, #x); ++bad; } } while (0)

// ---- the fake: page-locked memory of the current device; a reset of the device unlocks it ----
static int device = 0;
static std::map<void*, int> locked; // address -> device
static long locks = 0, unlocks = 0;
static bool none_left = false;
static cudaError_t last = cudaSuccess;

extern "C" {
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned)
{
    if (none_left) return last = cudaErrorMemoryAllocation;
    *p = std::malloc(bytes);
    std::memset(*p, 0xff, bytes);
    locked[*p] = device;
    ++locks;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p)
{
    CHECK(locked.erase(p) == 1);
    ++unlocks;
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned)
{
    *d = h;
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p)
{
    a->type = locked.count(const_cast<void*>(p)) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void)
{
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
}

namespace heomhost {
int set_error(int code, const std::string&) { return code; }
}

using heomrt::FlagPage;
using heomrt::HostFlag;

int main()
{
    // no page to be had: an error, and none of it left for the next launch's check
    none_left = true;
    {
        HostFlag f;
        CHECK(f.alloc(0) == HEOM_E_NOMEM && !f.page);
        CHECK(cudaGetLastError() == cudaSuccess);
    }
    none_left = false;

    // one handle after another: one page-lock for all of them
    for (int k = 0; k < 100; ++k) {
        HostFlag a, b;
        CHECK(a.alloc(0) == 0 && b.alloc(0) == 0);
        CHECK(a.dev != b.dev && !a.set() && !b.set());
        *a.dev = 1; // what a kernel does
        CHECK(a.set() && !b.set());
        a.clear();
        CHECK(!a.set());
        *a.dev = *b.dev = 1; // the next one's flags start clear all the same
    }
    CHECK(locks == 1 && unlocks == 0);

    // a page of its own for another device
    {
        HostFlag a, b;
        CHECK(a.alloc(0) == 0);
        device = 1;
        CHECK(b.alloc(1) == 0 && b.page != a.page && locked[b.page->host] == 1);
        device = 0;
        CHECK(locks == 2);
    }

    // a full page makes place for another and goes with its last flag; the newest page stays
    {
        const int more = FlagPage::kFlags + 10;
        std::unique_ptr<HostFlag[]> f(new HostFlag[more]);
        std::set<int*> seen;
        for (int k = 0; k < more; ++k) CHECK(f[k].alloc(0) == 0 && seen.insert(f[k].dev).second);
        CHECK(locks == 3 && f[0].page != f[more - 1].page);
    }
    CHECK(unlocks == 1);

    // a reset of the device takes its page along: the next handle gets a new one, and nobody frees the old one
    {
        HostFlag a;
        CHECK(a.alloc(0) == 0 && locks == 3);
        locked.erase(a.page->host);
        HostFlag b;
        CHECK(b.alloc(0) == 0 && locks == 4 && b.page != a.page);
    }
    CHECK(unlocks == 1);
    // the same when another's page-locked memory lies at the old address
    {
        HostFlag a;
        CHECK(a.alloc(0) == 0 && locks == 4);
        std::memset(a.page->host, 0, FlagPage::kMark * sizeof(int));
        HostFlag b;
        CHECK(b.alloc(0) == 0 && locks == 5 && b.page != a.page);
    }
    CHECK(unlocks == 1);

    // threads that make and drop handles: no two hold a flag at once
    std::atomic<int> owner[FlagPage::kFlags]{};
    {
        HostFlag keep;
        CHECK(keep.alloc(0) == 0);
        int* const base = keep.page->dev;
        std::vector<std::thread> t;
        for (int k = 0; k < 8; ++k)
            t.emplace_back([&] {
                for (int n = 0; n < 2000; ++n) {
                    HostFlag f;
                    CHECK(f.alloc(0) == 0);
                    CHECK(owner[f.dev - base].fetch_add(1) == 0);
                    owner[f.dev - base].fetch_sub(1);
                }
            });
        for (auto& x : t) x.join();
    }
    CHECK(locks == 5);
    printf("%s\n", bad ? "FAILED" : "ok");
    return bad ? 1 : 0;
}

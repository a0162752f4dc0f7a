// Host-only check of dm-heom_b200/csrc/device_memory.hpp over a fake of the CUDA calls that it makes (compiled by
// tests/test_device_memory.py).  Prints one line per problem, then "ok" or "FAILED".
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <set>
#include "device_memory.hpp"

static int bad = 0;
#define CHECK(x) \
    do { if (!(x)) { printf("bad line %d: %s\n", __LINE__, #x); ++bad; } } while (0)

// ---- the fake: host memory, and a number of calls after which there is none for a while ----
static long fail_from = -1, fail_count = 0, mallocs = 0;
static std::set<void*> live;
static cudaError_t last = cudaSuccess;

extern "C" {
cudaError_t cudaMalloc(void** p, size_t bytes)
{
    if (fail_from >= 0 && mallocs >= fail_from && mallocs < fail_from + fail_count) {
        ++mallocs;
        return last = cudaErrorMemoryAllocation;
    }
    ++mallocs;
    *p = std::malloc(bytes);
    live.insert(*p);
    return cudaSuccess;
}
cudaError_t cudaFree(void* p)
{
    CHECK(live.erase(p) == 1);
    std::free(p);
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

static void no_memory(long calls) // the next `calls` allocations fail
{
    fail_from = mallocs;
    fail_count = calls;
}

static void ring()
{
    heomrt::AdjointRing<double2> r;
    CHECK(r.resize(3, 40) && r.group == 3 && r.states.p && r.states.n == 120);
    const double2* at = r.states.p;
    CHECK(!r.resize(3, 40) && r.states.p == at);                  // nothing changed: captured sweeps stay valid
    CHECK(r.resize(2, 40) && r.group == 2 && r.states.p == at);   // a smaller group in the same memory
    // no memory for a larger one: the sweep goes on without a ring, and no error waits for the next launch's check
    no_memory(1);
    CHECK(r.resize(5, 40) && r.group == 0 && !r.states.p && r.states.n == 0);
    CHECK(cudaGetLastError() == cudaSuccess);
    // memory is back: the same request gets its ring
    CHECK(r.resize(5, 40) && r.group == 5 && r.states.p && r.states.n == 200);
    CHECK(r.resize(0, 40) && r.group == 0 && !r.states.p);
    CHECK(!r.resize(0, 40));
    no_memory(1);
    CHECK(!r.resize(4, 40) && r.group == 0 && !r.states.p);
    CHECK(r.resize(4, 40) && r.group == 4 && r.states.p);
}

static void buffers()
{
    heomrt::DevBuf<double> a, b;
    CHECK(a.ensure(100) == 0 && a.n == 100);
    const double* at = a.p;
    CHECK(a.ensure(60) == 0 && a.p == at && a.n == 100); // kept: what holds its address stays valid
    // no memory for a larger one: the buffer is empty and says so, and no error waits for the next launch's check
    no_memory(1);
    CHECK(a.ensure(200) == HEOM_E_NOMEM && !a.p && a.n == 0);
    CHECK(cudaGetLastError() == cudaSuccess);
    // the size it had before the failure is not there any more, and is asked for again
    const long before = mallocs;
    CHECK(a.ensure(60) == 0 && a.p && a.n == 60 && mallocs == before + 1);
    CHECK(b.ensure(5) == 0);
    a.swap(b);
    CHECK(a.n == 5 && b.n == 60 && a.p != b.p);
}

int main()
{
    buffers();
    ring();
    CHECK(live.empty());
    printf("%s\n", bad ? "FAILED" : "ok");
    return bad ? 1 : 0;
}

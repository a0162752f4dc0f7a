// A pipeline wait of the N <= 8 stage kernel that runs out (compiled and run by tests/test_gpu_wait.py).  The copies
// themselves arrive; chosen lanes overlook it.  With no H, bath term or same term the stage is
// out = in, so that what a warp wrote before it gave up can be told from what it did not.  Prints "bad ..." for any
// violation, then "ok" or "FAILED".
#include <cstdint>
#include <cstdio>
#include <vector>

// mode 0: every lane sees its copies arrive; 1: lane 5 never does; 2: no lane does; 3: lane 5 does not in its third
// wait (the first of the warp's two mbarriers, its second phase)
__constant__ int c_mode;
__device__ inline bool wait_seen(bool done, unsigned parity)
{
    const bool five = threadIdx.x % 32 == 5;
    return done && !(c_mode == 2 || (c_mode == 1 && five) || (c_mode == 3 && five && parity == 1));
}
#define HEOM_WAIT_SEEN(done, parity) wait_seen(done, parity)
#define HEOM_WAIT_TRIES (1 << 14)
#include "heom_kernels.cuh"
#include "row_tables.inc"

static int bad = 0;
#define TRY(x)                                                                         \
    do {                                                                               \
        const cudaError_t e_ = (x);                                                    \
        if (e_ != cudaSuccess) { printf("bad %s: %s\n", #x, cudaGetErrorString(e_)); ++bad; } \
    } while (0)

template <typename T>
T* upload(const std::vector<T>& v)
{
    T* p = nullptr;
    TRY(cudaMalloc(&p, v.size() * sizeof(T)));
    TRY(cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice));
    return p;
}

template <int N, int SLT>
void run(const char* name, void (*kernel)(const heomk::DmmaParams))
{
    constexpr int P = heomk::pairs_of(N), nodes = 45, blocks = 2, W = N * SLT, LS = 4;
    const int NW = (2 * W + 3) & ~3, TWB = (W + 15) & ~15, recb = heomk::rec_bytes(NW, TWB);
    std::vector<uint8_t> rec((size_t)nodes * recb, 0);
    for (int u = 0; u < nodes; ++u)
        for (int q = 0; q < NW; ++q) reinterpret_cast<int32_t*>(rec.data() + (size_t)u * recb)[q] = -1;
    std::vector<double2> in((size_t)nodes * 2 * P), mark(in.size(), make_double2(-7.0, -7.0));
    for (size_t q = 0; q < in.size(); ++q) in[q] = make_double2(1.0 + q, -0.5 * q);
    std::vector<int16_t> slots(N * SLT), pos(W);
    for (int q = 0; q < W; ++q) slots[q] = pos[q] = (int16_t)q;
    heomk::DmmaParams dp{};
    dp.p.in = upload(in);
    dp.p.out = upload(mark);
    dp.p.beta = make_double2(0.25, 0.0);
    dp.p.use_x = 1;
    dp.p.same_real = 1;
    dp.p.rec = upload(rec);
    dp.p.hfrag = upload(std::vector<double>(heomk::frag_doubles(N), 0.0));
    dp.p.gamma0 = upload(std::vector<double2>(N * N, make_double2(0.0, 0.0)));
    dp.p.slots = upload(slots);
    dp.p.nodes = nodes;
    dp.p.W = W;
    dp.p.NW = NW;
    dp.p.TWB = TWB;
    dp.p.LS = LS;
    dp.p.SL = SLT;
    for (int l = 0; l < 32; ++l)
        for (int s = 0; s < 2; ++s) {
            const int r = l >> 2, k = 2 * (l & 3) + s;
            dp.rt.pos[l][s] = -1;
            for (int p = 0; p < P; ++p)
                if (r < N && k < N && (kRowE1[N][p] == r * N + k || kRowE2[N][p] == r * N + k))
                    dp.rt.pos[l][s] = (signed char)p;
        }
    dp.ct.chat = upload(std::vector<double>(W, 0.0));
    dp.ct.khat = upload(std::vector<double2>(3 * W, make_double2(0.0, 0.0)));
    dp.ct.sq = upload(std::vector<double>(LS + 1, 1.0));
    dp.ct.pos = upload(pos);
    int* err = nullptr;
    TRY(cudaHostAlloc(&err, sizeof(int), cudaHostAllocMapped));
    TRY(cudaHostGetDevicePointer(&dp.err, err, 0));
    const size_t smem = heomk::dmma_smem_bytes(P, W, NW, TWB, LS);
    TRY(cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int warps = blocks * heomk::kRowWarps;
    for (int mode : {0, 1, 2, 3, 0}) {
        if (bad) return;
        TRY(cudaMemcpyToSymbol(c_mode, &mode, sizeof mode));
        TRY(cudaMemcpy(dp.p.out, mark.data(), mark.size() * 16, cudaMemcpyHostToDevice));
        *static_cast<volatile int*>(err) = 0;
        kernel<<<blocks, heomk::kRowWarps * 32, smem>>>(dp);
        TRY(cudaDeviceSynchronize());
        std::vector<double2> out(in.size());
        TRY(cudaMemcpy(out.data(), dp.p.out, out.size() * 16, cudaMemcpyDeviceToHost));
        const int want = mode == 0 ? 0 : 1;
        if (*static_cast<volatile int*>(err) != want) {
            printf("bad %s mode %d: flag %d\n", name, mode, *static_cast<volatile int*>(err));
            ++bad;
        }
        // a warp's ADOs written: all, none, or the two before its third wait
        const int done = mode == 0 ? nodes : mode == 3 ? 2 * warps : 0;
        for (int u = 0; u < nodes; ++u)
            for (int q = 0; q < 2 * P; ++q) {
                const double2 a = out[(size_t)u * 2 * P + q];
                const double2 b = u < done ? in[(size_t)u * 2 * P + q] : mark[0];
                if (a.x != b.x || a.y != b.y) {
                    printf("bad %s mode %d: ADO %d value %d is (%g, %g)\n", name, mode, u, q, a.x, a.y);
                    ++bad;
                    u = nodes;
                    break;
                }
            }
    }
}

int main()
{
    // one slot: a warp waits for an ADO when it starts on it, the next one's copies in flight; two: one ADO ahead
    run<4, 1>("one slot", heomk::heom_dmma_stage<4, heomk::H_REAL_SYM, 1, false, false, false>);
    run<4, 2>("two slots", heomk::heom_dmma_stage<4, heomk::H_REAL_SYM, 2, false, false, true>);
    printf("%s\n", bad ? "FAILED" : "ok");
    return bad ? 1 : 0;
}

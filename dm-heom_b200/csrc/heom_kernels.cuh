// heom_kernels.cuh -- sm_100a kernels of the HEOM derivative + RK4 path.
//
// heom_pair_stage evaluates the HEOM time derivative L(w) for every ADO of
// the hierarchy (the reference's heom_ode kernel,
// dm-heom/cl/heom/heom_ode.cl:24-451) and fuses the Runge-Kutta write of the
// stage into the same pass (the NOMA_NUM_ODE_ACCUMULATE /
// NOMA_NUM_ODE_SUBDIAGONAL write modes, heom_ode.cl:416-434, generalised to a
// complex stage coefficient).
//
// Per element (i, j) of ADO u the derivative is
//   L(w)_u(i,j) = i * sum_k [ w_u(i,k) Hs(k,j) - Hs(i,k) w_u(k,j) ]        (:89-114, Hs = H / hbar)
//               + (pf_same_sum[u] + gamma0(i,j)) w_u(i,j)                 (:131-168)
//               + sum over slots e = b*M+m of the baths b of site i:
//                    i cplus(n) w_{u+e}(i,j) + kappa_i(n) w_{u-e}(i,j)      (:183-221, :280-342)
//               + sum over slots e of the baths of site j:
//                   -i cplus(n) w_{u+e}(i,j) + kappa_j(n) w_{u-e}(i,j)      (:223-259, :344-403)
// with n the tuple entry of u for slot e and
//   cplus(n)   = sqrt((n+1) |c_e| / hbar)                                 (:211, :249)
//   kappa_i(n) = sqrt(n hbar / |c_e|) (i c_e / hbar + [m==0] pf_circ[b])  (:301-337)
//   kappa_j(n) = sqrt(n hbar / |c_e|) (-i c_e / hbar + [m==0] pf_circ[b]) (:363-398)
// For a diagonal element the site-i and site-j plus terms cancel exactly and
// the minus terms combine to kappa_i + kappa_j ("kappa_d"); both are folded
// on the host.
//
// HBM layout ("pair layout"): an ADO is P = N(N-1)/2 + ceil(N/2) sectors of
// 32 B.  Sector p < N(N-1)/2 holds the symmetric pair (w(i,j), w(j,i)), i < j;
// the remaining sectors hold pairs of diagonal elements (w(2k,2k),
// w(2k+1,2k+1)) (for odd N the last holds w(N-1,N-1) twice).  The neighbour
// terms only ever read the "cross" of a neighbour -- row b and column b for a
// bath b of the element's sites -- and in this layout a cross is N whole
// sectors; both elements of a sector need the same neighbours.  For N = 8 an
// ADO is exactly 32 sectors (1 KB): one warp per ADO, one sector per lane.
//
// Work mapping: N <= 8 one warp per ADO (heom_dmma_stage), N = 9..16 a team
// of TW = ceil(P/32) warps per ADO (heom_pair_stage); in both the commutator
// runs on the FP64 tensor pipe (m8n8k4) and the lane that owns a sector does
// its bath terms and the stage write.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace heomk {

constexpr int kCtaWarps = 8;
constexpr int kRowWarps = 4; // warps of a CTA of the N <= 8 stage kernel

__host__ __device__ constexpr int pairs_of(int n) { return n * (n - 1) / 2 + (n + 1) / 2; }
__host__ __device__ constexpr int team_warps(int n) { return (n * ((n + 1) / 2) + 31) / 32; }
__host__ __device__ constexpr int cta_teams(int n) { return team_warps(n) == 2 ? 2 : 1; }
__host__ __device__ constexpr int team_threads(int n) { return cta_teams(n) * team_warps(n) * 32; }

// element indices (row-major, e = i*N + j) of the two halves of sector p
__host__ __device__ inline void pair_elements(int n, int p, int* e1, int* e2, int* i_out, int* j_out,
                                              int* diag)
{
    const int noff = n * (n - 1) / 2;
    if (p < noff) {
        int i = 0, q = p;
        while (q >= n - 1 - i) {
            q -= n - 1 - i;
            ++i;
        }
        const int j = i + 1 + q;
        *e1 = i * n + j;
        *e2 = j * n + i;
        *i_out = i;
        *j_out = j;
        *diag = 0;
    } else {
        const int k = p - noff;
        const int a = 2 * k;
        const int b = (2 * k + 1 < n) ? 2 * k + 1 : a;
        *e1 = a * n + a;
        *e2 = b * n + b;
        *i_out = a;
        *j_out = b;
        *diag = 1;
    }
}

struct PairParams {
    const double2* __restrict__ in;  // [nodes][2P] (sector p = double2 pair 2p, 2p+1)
    const double2* y;                // AXPY against y instead of in (may alias out)
    double2* out;
    double2* acc;                    // accumulate mode
    double2 beta;                    // out = (use_x ? x : 0) + beta * L
    double2 acc_beta;                // acc = (acc_init ? in : acc) + acc_beta * L
    int use_x;
    int acc_init;
    int use_acc;
    int no_same;                     // leave out pf_same_sum (flow tracking)
    int same_real;                   // pf_same_sum and gamma0 are real
    // one record of rec_bytes(NW, TWB) per ADO: (plus, minus) of every slot as int32, padded to NW (multiple of 4);
    // the tuple bytes, padded to TWB (multiple of 16); pf_same_sum (double2)
    const unsigned char* __restrict__ rec;
    const double* __restrict__ hfrag;  // [n_inst][frag_doubles(N)] MMA operand fragments of H / hbar
    const int32_t* __restrict__ inst;  // [nodes] instance of each ADO; NULL when the handle holds one instance
    const double2* __restrict__ gamma0;// [N*N]
    const int16_t* __restrict__ slots; // [N][SL], -1 padded
    int64_t nodes;
    int W, NW, TWB, LS, SL;
};

enum HKind : int { H_REAL_SYM = 0, H_GENERIC = 1 };

__host__ __device__ constexpr int rec_bytes(int NW, int TWB) { return NW * 4 + TWB + 16; }

// MMA operand fragments of H / hbar, per instance: N <= 8 one 8 x 8 block and
// two k-slices, N = 9..16 a zero-padded 16 x 16 grid of 2 x 2 blocks and four
// k-slices.  Layout [kind][block b][k-slice s][lane], lane l = 4g + t:
// kind 0/1 = Re/Im of hb = H(c, 8b+g) (B operand of w H for block column b),
// kind 2/3 = Re/Im of ha = -H(8b+g, c) (A operand of -H w for block row b), c = frag_col(n, s, t).
__host__ __device__ constexpr int frag_blocks(int n) { return n <= 8 ? 1 : 2; }
__host__ __device__ constexpr int frag_slices(int n) { return n <= 8 ? 2 : 4; }
__host__ __device__ constexpr int frag_doubles(int n) { return 4 * frag_blocks(n) * frag_slices(n) * 32; }
// column (contraction index) of k-slice s in lane position t: N <= 8 the lane's own columns 2t, 2t+1
__host__ __device__ constexpr int frag_col(int n, int s, int t) { return n <= 8 ? 2 * t + s : 4 * s + t; }
__host__ __device__ constexpr int frag_index(int n, int kind, int b, int s, int lane)
{
    return ((kind * frag_blocks(n) + b) * frag_slices(n) + s) * 32 + lane;
}

// Team kernel (N = 9..16): the staged ADO is row-major with row stride
// TS = 4 (mod 8) double2 and the columns of rows with bit 1 set swapped in
// pairs (k ^ 2), so that the quarter-warp reads of both MMA operands,
// A = w(8I+g, 4s+t) and B = w(4s+t, 8J+g), hit eight distinct 16-byte bank groups.
__host__ __device__ constexpr int tile_stride(int n) { return (n + 3) / 8 * 8 + 4; }
__host__ __device__ constexpr int tile_pos(int n, int i, int k) { return i * tile_stride(n) + (k ^ (i & 2)); }
// exchange tile of the commutator: 16 rows of 17 double2 (conflict-free C writes)
constexpr int kXchStride = 17;
constexpr int kXchBytes = 16 * kXchStride * 16;

// shared look-up tables of the stage kernels: khat 3*W double2, (sqrt(n),
// sqrt(n+1)) LS+1 double2, chat W doubles; padded to 128 bytes, since the tiles
// of the lockstep kernel follow: off a 32-byte boundary they cost 4 to 6 % (256
// instances of 7 states, depth 6: 217 -> 226 us a stage; 128 of 8, depth 5: 98.7
// -> 105.3; on a 128-byte boundary 219.8 and 97.2)
__host__ __device__ inline int dmma_lut_bytes(int W, int LS)
{
    return ((3 * W * 16 + (LS + 1) * 16 + W * 8) + 127) & ~127;
}

// dynamic shared memory carve-up (bytes); everything 16-B aligned
struct PairSmem {
    int lut;     // coefficient tables (dmma_lut_bytes)
    int team;    // per team: 2 slots, 2 exchange tiles, the hand-over buffers, gamma0
    int slot;    // per slot: tile + nbr + tup + pss
    int tile_off, nbr_off, tup_off, pss_off, xch_off;
    int hand_off, gam_off; // terms handed over (two copies of [2][threads]), gamma0 of the owned elements
};

__host__ __device__ inline PairSmem pair_smem_layout(int n, int W, int NW, int TWB, int LS)
{
    PairSmem s;
    s.lut = dmma_lut_bytes(W, LS);
    const int tile = n * tile_stride(n) * 16;
    s.tile_off = 0;
    s.nbr_off = tile;
    s.tup_off = s.nbr_off + ((NW * 4 + 15) & ~15);
    s.pss_off = s.tup_off + ((TWB + 15) & ~15);
    s.slot = s.pss_off + 16;
    s.xch_off = 2 * s.slot;
    s.hand_off = s.xch_off + 2 * kXchBytes;
    s.gam_off = s.hand_off + 2 * 2 * team_warps(n) * 32 * 16;
    s.team = s.gam_off + 2 * team_warps(n) * 32 * 16;
    return s;
}

__host__ inline size_t pair_smem_bytes(int n, int W, int NW, int TWB, int LS)
{
    const PairSmem s = pair_smem_layout(n, W, NW, TWB, LS);
    return (size_t)s.lut + (size_t)cta_teams(n) * s.team;
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

template <int TW>
__device__ __forceinline__ void team_sync(int team)
{
    if (TW == 1) {
        __syncwarp();
    } else {
        asm volatile("bar.sync %0, %1;\n" ::"r"(team + 1), "r"(TW * 32) : "memory");
    }
}

__device__ __forceinline__ void cmac(double2& acc, const double2 a, const double2 b)
{
    acc.x = fma(a.x, b.x, acc.x);
    acc.x = fma(-a.y, b.y, acc.x);
    acc.y = fma(a.x, b.y, acc.y);
    acc.y = fma(a.y, b.x, acc.y);
}

// ---------------------------------------------------------------------------
// N <= 8: one warp per ADO, one lane per (state, column pair).
//
// Lane 4r + t works for state r and the columns 2t, 2t+1 (the tile is
// zero-padded to 8 x 8): it holds the sectors of the pairs {r, 2t} and
// {r, 2t+1} (for t = r / 2 the diagonal sector stands for {r, r}).
//   * Commutator on the FP64 tensor pipe: the row elements (r, 2t+s) are the A
//     fragment of w H and the column elements (2t+s, r) the B fragment of H w
//     for k-slice s (k = 2t + s), and the C fragment is (r, 2t), (r, 2t+1):
//     the lane's own row elements.  Eight m8n8k4 MMAs for real H, sixteen for
//     complex H.
//   * Bath terms: the lane reads its two sectors of the neighbours along the
//     baths of state r only, so the slot's index, sqrt(n) and coefficients are
//     looked up once for four elements.  They give the row-r terms of the row
//     elements and the column-r terms of the column elements.
//   * A sector {r, c} is held by a lane of row r and a lane of row c.  One of
//     them owns it (row_owned); the other hands over its terms by eight
//     shuffles, and the owner writes the 32-byte sector.  A sector's first
//     half is the owner's row element, so that all coefficients are in place.
//
// Pipeline: per warp two slots, each filled by two 1-D TMA bulk copies (tile,
// record) that complete on the slot's mbarrier; the copies of ADO k+1 fly
// while ADO k is computed.  Every wait is bounded.  The MMAs and shuffles are the
// whole warp's work, so if the wait of a lane expires the warp leaves as a whole:
// where it waits for the next ADO (two slots and more) once this one is done, else
// at once.  It then waits, bounded again, for the copies in flight and sets *err.
//
// What bounds it: the L1 data pipe (8 states, two slots, 245,157 ADOs: 135
// wavefronts in 201 cycles per ADO and SM, 75 of them shared memory) and the
// latency of 20 warps per SM; on 735,471 ADOs, a state beyond L2, DRAM is the
// nearer limit (1.84 x the algorithmic bytes).  Measured against a lane per
// sector, which looked up both sites' slots for two elements (us per stage, one
// B200): 8 states, two slots, 735,471
// ADOs 791 -> 547, 74,613 ADOs 76.0 -> 51.8; one slot, 24,310 ADOs 21.5 -> 14.9,
// 319,770 ADOs 235 -> 217; 7 states, one slot, 6435 ADOs 9.75 -> 6.6; 330 ADOs
// 4.6 -> 3.1 (mostly the dependent launch).  503 -> 352 instructions and 204 ->
// 135 wavefronts per ADO; most of the fewer are shared memory's (130 -> 75), the
// rest a store that is linear in the lanes (22 -> 8) and owned sectors side by side.
// A lane table read from the parameter bank has to be held (opaque): reloaded
// under register pressure it cost 180 instructions per ADO and half the speed.
// Two slots: the K neighbours are read one ADO ahead and the coefficients come
// from shared memory (in registers they spill: 1137 us); one slot: the other
// way round.  Two slots: reading the real parts of the same term's factors alone
// and the own sector's halves in a staggered order took 13 wavefronts more:
// 74,613 ADOs 50.1, 735,471 ADOs 540.  The votes by which a warp leaves as a whole
// cost 0.4 % (74,613 ADOs 50.35), 6435 ADOs of 7 states 1.5 % (6.31 -> 6.40); with
// the vote in every lane's way to its loads 74,613 ADOs took 51.0.
// ---------------------------------------------------------------------------

// which of its two sectors lane (r, t) owns: 0 = {r, 2t}, 1 = {r, 2t+1}
__host__ __device__ constexpr int row_owned(int r, int t)
{
    return t == (r >> 1) ? 0 : (r & 1) ^ ((r >> 1) > t ? 1 : 0);
}

// sector position of pair {r, 2t+s} for lane 4r + t (-1: outside N x N)
struct RowTab {
    signed char pos[32][2];
};

// lane tables of the lockstep kernel: the operand sectors of every lane and
// which half holds the row element.  A lane outside N x N has those of a lane
// of its quarter warp that is inside and not on the diagonal (where there is one).
struct LaneTab {
    signed char e1[32], e2[32]; // sector of lane p: element indices (row-major)
    signed char ord[32];        // the sectors in the order in which the warps take them
    signed char fs[32][2];      // operand sector of k-slice s
    signed char ha[32][2];      // half of that sector holding A = w(r, 2t+s)
};

// Factored bath coefficients: cplus(n) = chat * sqrt(n+1), kappa(n) = khat * sqrt(n)
// (heom_ode.cl:211,249 and :321,383).  Per-slot constants are stored at
// position pos(slot) = m * B + b (slot = b*M + m) so that the lanes of a warp,
// which read the same m for different baths, hit different banks.
struct CoefTabs {
    const double* chat;   // [W] at pos(slot)
    const double2* khat;  // [3][W] at pos(slot): kappa_i, kappa_j, kappa_i + kappa_j (n = 1)
    const double* sq;     // [D+2]: sqrt(n)
    const int16_t* pos;   // [W] slot -> position
};

struct DmmaParams {
    PairParams p;
    RowTab rt; // N <= 8
    CoefTabs ct;
    int* err; // mapped host memory
};

__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(c0), "+d"(c1)
                 : "d"(a), "d"(b));
}

// 32 bytes through the coherent path: a stage runs as a dependent of the kernel that writes what it reads
__device__ __forceinline__ void ld256(const double2* src, double2& a, double2& b)
{
    asm volatile("ld.global.v4.f64 {%0,%1,%2,%3}, [%4];\n"
                 : "=d"(a.x), "=d"(a.y), "=d"(b.x), "=d"(b.y)
                 : "l"(src));
}

// 32-byte stores when ok, without a branch (streaming / default cache policy)
__device__ __forceinline__ void st256_cs_if(bool ok, double2* dst, double2 a, double2 b)
{
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %5, 0;\n @q st.global.cs.v4.f64 [%0], {%1,%2,%3,%4};\n}\n" ::"l"(dst),
                 "d"(a.x), "d"(a.y), "d"(b.x), "d"(b.y), "r"((unsigned)ok)
                 : "memory");
}
__device__ __forceinline__ void st256_if(bool ok, double2* dst, double2 a, double2 b)
{
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %5, 0;\n @q st.global.v4.f64 [%0], {%1,%2,%3,%4};\n}\n" ::"l"(dst),
                 "d"(a.x), "d"(a.y), "d"(b.x), "d"(b.y), "r"((unsigned)ok)
                 : "memory");
}

__device__ __forceinline__ void st256_cs(double2* dst, double2 a, double2 b)
{
    asm volatile("st.global.cs.v4.f64 [%0], {%1,%2,%3,%4};\n" ::"l"(dst), "d"(a.x), "d"(a.y), "d"(b.x),
                 "d"(b.y)
                 : "memory");
}

__device__ __forceinline__ void st256(double2* dst, double2 a, double2 b)
{
    asm volatile("st.global.v4.f64 [%0], {%1,%2,%3,%4};\n" ::"l"(dst), "d"(a.x), "d"(a.y), "d"(b.x), "d"(b.y)
                 : "memory");
}

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_addr(bar)) : "memory");
}

__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes, uint64_t* bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}

__device__ __forceinline__ void mbar_expect(uint64_t* bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}

// tries of a bounded wait (a second or so) and what a lane makes of one: a test may have chosen lanes overlook that
// the phase is complete, with fewer tries
#ifndef HEOM_WAIT_TRIES
#define HEOM_WAIT_TRIES (1 << 24)
#endif
#ifndef HEOM_WAIT_SEEN
#define HEOM_WAIT_SEEN(done, parity) (done)
#endif

__device__ __forceinline__ bool mbar_try(uint64_t* bar, unsigned parity)
{
    unsigned done;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                 " selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(done)
                 : "r"(smem_addr(bar)), "r"(parity)
                 : "memory");
    return done != 0;
}

// bounded wait of a lane for the phase `parity` of an mbarrier; false on expiry
__device__ __forceinline__ bool lane_wait(uint64_t* bar, unsigned parity)
{
    for (int it = 0; it < HEOM_WAIT_TRIES; ++it)
        if (HEOM_WAIT_SEEN(mbar_try(bar, parity), parity)) return true;
    return false;
}

// the same of a whole warp, with one answer for every lane
__device__ __forceinline__ bool warp_wait(uint64_t* bar, unsigned parity)
{
    for (int it = 0; it < HEOM_WAIT_TRIES; ++it)
        if (__all_sync(0xffffffffu, HEOM_WAIT_SEEN(mbar_try(bar, parity), parity))) return true;
    return false;
}

// the time of a wait for copies that nothing is done with any more
__device__ __forceinline__ void drain(uint64_t* bar, unsigned parity)
{
    for (int it = 0; it < HEOM_WAIT_TRIES && !mbar_try(bar, parity); ++it) {
    }
}

// bytes of one pipeline slot and of a warp's shared area for the DMMA kernel:
// the tile, the ADO's record and 16 bytes of zeros (operands outside N x N)
__host__ __device__ inline int dmma_slot_bytes(int P, int NW, int TWB)
{
    return P * 32 + ((rec_bytes(NW, TWB) + 15) & ~15) + 16;
}
__host__ __device__ inline int dmma_warp_bytes(int P, int NW, int TWB)
{
    return 2 * dmma_slot_bytes(P, NW, TWB) + 16 /* 2 mbarriers */;
}
__host__ inline size_t dmma_smem_bytes(int P, int W, int NW, int TWB, int LS)
{
    return (size_t)dmma_lut_bytes(W, LS) + 2 * 32 * 16 + (size_t)kRowWarps * dmma_warp_bytes(P, NW, TWB);
}

// 32 bytes at src when v >= 0; otherwise a and b keep what they hold
__device__ __forceinline__ void ld256_if(int v, const double2* src, double2& a, double2& b)
{
    asm volatile("{\n .reg .pred q;\n setp.ge.s32 q, %5, 0;\n @q ld.global.v4.f64 {%0,%1,%2,%3}, [%4];\n}\n"
                 : "+d"(a.x), "+d"(a.y), "+d"(b.x), "+d"(b.y)
                 : "l"(src), "r"(v));
}

__device__ __forceinline__ double2 shfl2(double2 v, int src)
{
    return make_double2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}
__device__ __forceinline__ double2 sel2(bool q, double2 a, double2 b)
{
    return make_double2(q ? a.x : b.x, q ? a.y : b.y);
}

// a value the compiler has to keep: under register pressure it otherwise loads a lane's table entry from the
// parameter bank again and again, and a constant load with 32 different addresses takes 32 turns
__device__ __forceinline__ int opaque(int v)
{
    asm volatile("" : "+r"(v));
    return v;
}

// dependent launch: the next kernel of the stream may start its prologue; wait
// until the kernels before this one are complete and their writes visible
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

// CTAs of four warps per SM. Two slots: five (96 registers a thread, 20 warps; 8 states, 735,471 ADOs: 547 us a
// stage, against 608 at 16 warps and 789 at 24 with 56 bytes spilled). One slot: four (8 states, 24,310 ADOs 14.9
// us, 7 states, 6435 ADOs 6.6; five spill a little: 15.4 and 7.0, and gain only far beyond L2, 319,770 ADOs 211 us
// against 217). Complex H, batches and more slots need the registers.
constexpr int row_blocks(int hk, int slt, bool mi) { return hk == H_REAL_SYM && slt == 2 && !mi ? 5 : 4; }

// MI: the handle holds several instances (p.inst set); each ADO's instance
// selects its H fragments, reloaded whenever the instance changes.
// ADJ: apply the adjoint operator L^H instead of L.  The caller passes the
// tables of -H^H (fragments) and conj(gamma0); pf_same_sum is conjugated here.
// In the bath terms the roles of the neighbours swap: the plus neighbour enters
// with conj(khat) sqrt(n+1), the minus neighbour with -/+ i chat sqrt(n).
// "K" is the neighbour with the complex coefficient (minus for L, plus for
// L^H), "C" the one with the imaginary coefficient.
// GEN: every write mode; otherwise out = in + beta L only (the product form), whose
// epilogue tests no mode and holds no pointer for one.  us per stage of the product
// form through the first / the second: 8 states, two slots, 74,613 ADOs 52.2 / 50.7,
// 735,471 ADOs 552 / 545; one slot, 24,310 ADOs 15.9 / 15.2; 7 states, one slot, 6435
// ADOs 6.60 / 6.24; 4 states, three slots, 18,564 ADOs 18.5 / 17.4; 6 states, one
// slot, 8008 ADOs 7.22 / 7.18.
template <int N, int HK, int SLT, bool MI, bool ADJ, bool GEN>
__global__ void __launch_bounds__(kRowWarps * 32, row_blocks(HK, SLT, MI)) heom_dmma_stage(const __grid_constant__ DmmaParams dp)
{
    static_assert(N <= 8, "DMMA stage handles N <= 8");
    constexpr int P = pairs_of(N);
    constexpr bool AHEAD = SLT > 1;            // read the K neighbours one ADO ahead
    constexpr bool XLATE = SLT > 1;            // read the sector's own values again at the end
    constexpr bool SPLIT = SLT > 1;            // same term: real parts first (one slot: the split spills)
    constexpr bool KREG = SLT == 1;            // coefficients in registers (two slots: they would spill)
    constexpr int QB = SLT < 2 ? SLT : 2;      // slots whose neighbours are read in one batch
    constexpr bool ODD = (N & 1) != 0;         // some lanes hold one sector only
    constexpr unsigned tile_b = P * 32;
    const PairParams& p = dp.p;
    extern __shared__ __align__(128) unsigned char smem[];
    const int W = p.W, LS = p.LS, SL = p.SL;

    grid_launch_dependents();
    double2* s_kh = reinterpret_cast<double2*>(smem);            // [3][W]: kappa_i, kappa_j, kappa_i + kappa_j
    double2* s_sq = s_kh + 3 * W;                                 // LS + 1: (sqrt(n), sqrt(n+1))
    double* s_ch = reinterpret_cast<double*>(s_sq + LS + 1);      // W
    for (int q = threadIdx.x; q < 3 * W; q += blockDim.x) s_kh[q] = dp.ct.khat[q];
    for (int q = threadIdx.x; q < W; q += blockDim.x) s_ch[q] = dp.ct.chat[q];
    for (int q = threadIdx.x; q <= LS; q += blockDim.x)
        s_sq[q] = make_double2(dp.ct.sq[q], q < LS ? dp.ct.sq[q + 1] : 0.0);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int slot_b = dmma_slot_bytes(P, p.NW, p.TWB);
    const unsigned recb = rec_bytes(p.NW, p.TWB);
    // per warp: the two mbarriers, then the two slots (tile, record, zeros)
    double2* s_g0 = reinterpret_cast<double2*>(smem + dmma_lut_bytes(W, LS));
    unsigned char* wbase = smem + dmma_lut_bytes(W, LS) + 1024 + warp * dmma_warp_bytes(P, p.NW, p.TWB);
    uint64_t* bars = reinterpret_cast<uint64_t*>(wbase);
    unsigned char* slot = wbase + 16;           // slot of the current ADO
    unsigned char* slot_n = slot + slot_b;      // slot of the next one
    const int tup_off = tile_b + p.NW * 4;
    const int pss_off = tup_off + p.TWB;

    // ---- this lane's place ----
    const int r = lane >> 2, t = lane & 3;
    const bool odd = row_owned(r, t) != 0;              // owns {r, 2t+1}
    const bool dga = t == (r >> 1) && !(r & 1);         // its sector 0 is the diagonal one (owned)
    const bool dgb = t == (r >> 1) && (r & 1);          // its sector 1 is the diagonal one (handed over)
    const int ps0 = opaque(dp.rt.pos[lane][0]), ps1 = opaque(dp.rt.pos[lane][1]);
    const int pso = odd ? ps1 : ps0, psg = odd ? ps0 : ps1; // owned, handed over
    const bool owner = pso >= 0, holds = psg >= 0;
    // the lane that hands over this lane's owned sector
    const int giver = t == (r >> 1) ? lane ^ 4 : 4 * (2 * t + (odd ? 1 : 0)) + (r >> 1);
    // operand offsets in a slot (bytes): row and column element of both sectors
    const int zero_off = slot_b - 16;
    const int ro0 = ps0 >= 0 ? ps0 * 32 + (odd ? 16 : 0) : zero_off;
    const int co0 = ps0 >= 0 ? ps0 * 32 + (odd ? 0 : 16) : zero_off; // diagonal: the second diagonal element
    const int ro1 = ps1 >= 0 ? ps1 * 32 + (odd ? 0 : 16) : zero_off;
    const int co1 = ps1 >= 0 ? (dgb ? ro1 : ps1 * 32 + (odd ? 16 : 0)) : zero_off;
    // negative: no such sector; no C term on it (diagonal)
    const int no_o = owner ? 0 : -1, no_g = holds ? 0 : -1;
    const int no_co = dga ? -1 : no_o, no_cg = dgb ? -1 : no_g;
    const double2* in_o = p.in + 2 * (owner ? pso : 0);
    const double2* in_g = p.in + 2 * (holds ? psg : 0);
    const int xh = (pso & 4) ? 16 : 0; // which half of its own sector a lane reads first (conflict-free quarter warps)

    // gamma0 of the lane's row elements ([2][32], the same for every warp)
    // SPLIT: the real parts of both, then the imaginary parts, which are read only where a bath has some
    if (warp < 2) {
        const double2 z = make_double2(0.0, 0.0);
        const double2 e0 = ps0 >= 0 ? p.gamma0[r * N + 2 * t] : z, e1 = ps1 >= 0 ? p.gamma0[r * N + 2 * t + 1] : z;
        s_g0[threadIdx.x] = SPLIT ? (warp ? make_double2(e0.y, e1.y) : make_double2(e0.x, e1.x)) : (warp ? e1 : e0);
    }
    int slo[SLT];                                       // record offsets of the slots of state r: their tuple byte
    int kp[SLT];                                        // table positions of the slots (-1: none)
    double2 kof[SLT], kgs[SLT], kj[SLT];                // KREG: coefficients of the row elements, of the column elements
#pragma unroll
    for (int q = 0; q < SLT; ++q) {
        const int sl = (r < N && q < SL) ? p.slots[r * SL + q] : -1;
        slo[q] = sl >= 0 ? sl : 0;
        kp[q] = sl >= 0 ? dp.ct.pos[sl] : -1;
        if (KREG) {
            const double2* k = dp.ct.khat + kp[q];
            const double2 z = make_double2(0.0, 0.0);
            kof[q] = sl >= 0 ? k[dga ? 2 * W : 0] : z;
            kgs[q] = sl >= 0 ? k[dgb ? 2 * W : 0] : z;
            kj[q] = sl >= 0 ? k[W] : z;
            if (ADJ) {
                kof[q].y = -kof[q].y;
                kgs[q].y = -kgs[q].y;
                kj[q].y = -kj[q].y;
            }
        }
    }
    const double2* kt_of = s_kh + (dga ? 2 : 0) * W;
    const double2* kt_gs = s_kh + (dgb ? 2 : 0) * W;
    const double2* kt_j = s_kh + W;

    if (lane == 0) {
        mbar_init(&bars[0]);
        mbar_init(&bars[1]);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (lane < 2) *reinterpret_cast<double2*>(slot + lane * slot_b + zero_off) = make_double2(0.0, 0.0);
    __syncthreads();

    const unsigned nodes = (unsigned)p.nodes; // at most 2^31 - 1
    const unsigned stride = gridDim.x * kRowWarps;
    unsigned u = blockIdx.x * kRowWarps + warp;
    // instance of the current ADO (warp-uniform); its fragments are in hb_* / ha_*
    int ci = (MI && u < nodes) ? __ldg(p.inst + u) : 0;
    // the next ADO's instance, read one iteration ahead of its use so that the
    // instance compare never waits on the load
    int ni_ahead = (MI && u + stride < nodes) ? __ldg(p.inst + u + stride) : ci;

    grid_wait(); // the state and the H tables of a field are written by the kernels before this one

    // operand fragments of H / hbar for k-slice s, k = 2t + s (zero outside the N x N block):
    //   hb = H(k, r) (B operand of w H), ha = -H(r, k) (A operand of -H w);
    // packed per instance as [re hb s0, s1 | im hb | re ha | im ha][lane]
    double hb_r[2], hb_i[2], ha_r[2], ha_i[2];
    auto load_frag = [&](int c, double* br, double* bi, double* ar, double* ai) {
        const double* f = dp.p.hfrag + (size_t)c * 256 + lane;
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            br[s] = f[32 * s];
            if (HK == H_GENERIC) {
                ar[s] = f[32 * (4 + s)];
                bi[s] = f[32 * (2 + s)];
                ai[s] = f[32 * (6 + s)];
            } else {
                ar[s] = bi[s] = ai[s] = 0.0;
            }
        }
    };
    load_frag(ci, hb_r, hb_i, ha_r, ha_i);

    auto issue = [&](unsigned v, unsigned char* dst, uint64_t* bar) {
        mbar_expect(bar, tile_b + recb);
        bulk_g2s(dst, p.in + (int64_t)v * (2 * P), tile_b, bar);
        bulk_g2s(dst + tile_b, p.rec + (int64_t)v * recb, recb, bar);
    };
    // the neighbours of the first slots' batch (QB slots) are read one ADO ahead: vk, vc their indices along K and C,
    // xo, xg the K neighbours' sectors
    int vk[QB], vc[QB];
    double2 xo[QB][2], xg[QB][2];
    auto load_k = [&](const unsigned char* sl, int q0) {
        const int2* nb = reinterpret_cast<const int2*>(sl + tile_b);
#pragma unroll
        for (int b = 0; b < QB; ++b) {
            const int2 pm = kp[q0 + b] >= 0 ? nb[slo[q0 + b]] : make_int2(-1, -1);
            vk[b] = ADJ ? pm.x : pm.y;
            vc[b] = ADJ ? pm.y : pm.x;
            const int64_t o = (int64_t)vk[b] * (2 * P);
            ld256_if(ODD ? vk[b] | no_o : vk[b], in_o + o, xo[b][0], xo[b][1]);
            ld256_if(ODD ? vk[b] | no_g : vk[b], in_g + o, xg[b][0], xg[b][1]);
        }
    };
    unsigned it = 0; // ADOs done: slot it & 1, mbarrier parity (it >> 1) & 1
    bool failed = false;
    if (u < nodes) {
        if (lane == 0) issue(u, slot, bars);
        if (AHEAD) {
            if (warp_wait(bars, 0)) load_k(slot, 0);
            else failed = true;
        }
    }
    for (; u < nodes && !failed; u += stride, ++it) {
        const bool more = u + stride < nodes;
        // (the slot's last readers are behind the __syncwarp of the previous iteration)
        if (more && lane == 0) issue(u + stride, slot_n, bars + ((it & 1) ^ 1));
        // the next ADO's instance and, when it differs, its fragments (used from the next iteration)
        int ni = ci;
        double nb_r[2], nb_i[2], na_r[2], na_i[2];
        if (MI && more) {
            ni = ni_ahead;
            if (ni != ci) load_frag(ni, nb_r, nb_i, na_r, na_i);
            ni_ahead = u + 2 * stride < nodes ? __ldg(p.inst + u + 2 * stride) : ni;
        }
        if (!AHEAD) {
            if (!warp_wait(bars + (it & 1), (it >> 1) & 1)) {
                failed = true;
                break;
            }
            load_k(slot, 0);
        }
        const unsigned char* tu = slot + tup_off;

        // ---- commutator on the tensor pipe, same term ----
        double2 of, os, gf, gs; // owned / handed-over sector, first / second half
        double2 xf, xs;         // the owned sector's own values
        {
            const double2 r0 = *reinterpret_cast<const double2*>(slot + ro0);
            const double2 c0 = *reinterpret_cast<const double2*>(slot + co0);
            const double2 r1 = *reinterpret_cast<const double2*>(slot + ro1);
            const double2 c1 = *reinterpret_cast<const double2*>(slot + co1);
            double2 pss = *reinterpret_cast<const double2*>(slot + pss_off);
            if (GEN && p.no_same) pss = make_double2(0.0, 0.0);
            if (ADJ) pss.y = -pss.y;
            if (!XLATE) {
                xf = sel2(odd, r1, r0);
                xs = sel2(odd, c1, c0);
            }
            double cr0 = 0.0, cr1 = 0.0, ci0 = 0.0, ci1 = 0.0;
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                const double2 A = s ? r1 : r0;
                const double2 B = s ? c1 : sel2(dga, r0, c0);
                dmma(cr0, cr1, A.x, hb_r[s]); // Re(w) Re(H)
                dmma(ci0, ci1, A.y, hb_r[s]); // Im(w) Re(H)
                if (HK == H_GENERIC) {
                    dmma(cr0, cr1, ha_r[s], B.x);  // -Re(H) Re(w)
                    dmma(ci0, ci1, ha_r[s], B.y);  // -Re(H) Im(w)
                    dmma(cr0, cr1, -A.y, hb_i[s]); // -Im(w) Im(H)
                    dmma(ci0, ci1, A.x, hb_i[s]);  //  Re(w) Im(H)
                    dmma(cr0, cr1, -ha_i[s], B.y); // +Im(H) Im(w)
                    dmma(ci0, ci1, ha_i[s], B.x);  // -Im(H) Re(w)
                } else { // H(r, k) = H(k, r): the fragment of w H serves both products
                    dmma(cr0, cr1, hb_r[s], -B.x);
                    dmma(ci0, ci1, hb_r[s], -B.y);
                }
            }
            // row elements: i * (w H - H w) / hbar and the same term
            double2 t0 = make_double2(-ci0, cr0), t1 = make_double2(-ci1, cr1);
            if (SPLIT) {
                const double2 gr = s_g0[lane];
                const double s0 = pss.x + gr.x, s1 = pss.x + gr.y;
                t0.x = fma(s0, r0.x, t0.x);
                t0.y = fma(s0, r0.y, t0.y);
                t1.x = fma(s1, r1.x, t1.x);
                t1.y = fma(s1, r1.y, t1.y);
                if (!p.same_real) {
                    const double2 gi = s_g0[32 + lane];
                    const double u0 = pss.y + gi.x, u1 = pss.y + gi.y;
                    t0.x = fma(-u0, r0.y, t0.x);
                    t0.y = fma(u0, r0.x, t0.y);
                    t1.x = fma(-u1, r1.y, t1.x);
                    t1.y = fma(u1, r1.x, t1.y);
                }
            } else {
                const double2 g0 = s_g0[lane], g1 = s_g0[32 + lane];
                cmac(t0, make_double2(pss.x + g0.x, pss.y + g0.y), r0);
                cmac(t1, make_double2(pss.x + g1.x, pss.y + g1.y), r1);
            }
            of = sel2(odd, t1, t0);
            gs = sel2(odd, t0, t1);
            os = gf = make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int q0 = 0; q0 < SLT; q0 += QB) {
            if (q0 > 0) load_k(slot, q0);
            // ---- bath terms: K neighbours ----
#pragma unroll
            for (int b = 0; b < QB; ++b) {
                const int q = q0 + b;
                if (vk[b] >= 0) {
                    const double2* sq = s_sq + tu[slo[q]];
                    const double sk = ADJ ? sq->y : sq->x;
                    auto kap = [&](const double2& reg, const double2* tab) {
                        const double2 v = KREG ? reg : tab[kp[q]];
                        return make_double2(v.x * sk, (ADJ && !KREG ? -v.y : v.y) * sk);
                    };
                    cmac(of, kap(kof[q], kt_of), xo[b][0]);
                    cmac(gs, kap(kgs[q], kt_gs), xg[b][1]);
                    const double2 k = kap(kj[q], kt_j);
                    if (!dga) cmac(os, k, xo[b][1]);
                    if (!dgb) cmac(gf, k, xg[b][0]);
                }
            }
            // ---- C neighbours (a diagonal element's terms of its row and column cancel) ----
#pragma unroll
            for (int b = 0; b < QB; ++b) {
                const int64_t o = (int64_t)vc[b] * (2 * P);
                if (vc[b] >= 0) {
                    ld256_if(no_co, in_o + o, xo[b][0], xo[b][1]);
                    ld256_if(no_cg, in_g + o, xg[b][0], xg[b][1]);
                }
            }
#pragma unroll
            for (int b = 0; b < QB; ++b) {
                const int q = q0 + b;
                if (vc[b] >= 0) {
                    const double2 sq = s_sq[tu[slo[q]]];
                    const double c = ADJ ? -s_ch[kp[q]] * sq.x : s_ch[kp[q]] * sq.y;
                    if (!dga) {
                        of.x = fma(-c, xo[b][0].y, of.x);
                        of.y = fma(c, xo[b][0].x, of.y);
                        os.x = fma(c, xo[b][1].y, os.x);
                        os.y = fma(-c, xo[b][1].x, os.y);
                    }
                    if (!dgb) {
                        gf.x = fma(c, xg[b][0].y, gf.x);
                        gf.y = fma(-c, xg[b][0].x, gf.y);
                        gs.x = fma(-c, xg[b][1].y, gs.x);
                        gs.y = fma(c, xg[b][1].x, gs.y);
                    }
                }
            }
        }
        // ---- the next ADO's K neighbours: in flight through the exchange, the stores and its commutator ----
        if (AHEAD && more) {
            if (lane_wait(bars + ((it & 1) ^ 1), ((it + 1) >> 1) & 1)) load_k(slot_n, 0);
            else failed = true; // (the warp leaves as a whole, after this ADO)
        }
        // ---- the handed-over sector's terms to its owner ----
        const double2 hf = shfl2(gf, giver), hs = shfl2(gs, giver);
        const double2 L1 = make_double2(of.x + hf.x, of.y + hf.y);
        double2 L2 = make_double2(os.x + hs.x, os.y + hs.y);
        if (ODD && r == N - 1 && dga) L2 = L1; // the padding half mirrors its element

        if (owner) {
            const int64_t off = (int64_t)u * (2 * P) + 2 * pso;
            if (XLATE) {
                const double2 xa = *reinterpret_cast<const double2*>(slot + pso * 32 + xh);
                const double2 xb = *reinterpret_cast<const double2*>(slot + pso * 32 + (xh ^ 16));
                xf = sel2(xh == 0, xa, xb);
                xs = sel2(xh == 0, xb, xa);
            }
            double2 o1 = xf, o2 = xs;
            if (GEN) {
                if (p.y) ld256(p.y + off, o1, o2);
                if (!p.use_x) o1 = o2 = make_double2(0.0, 0.0);
            }
            cmac(o1, p.beta, L1);
            cmac(o2, p.beta, L2);
            st256_cs(p.out + off, o1, o2);
            if (GEN && p.use_acc) {
                double2 a1 = xf, a2 = xs;
                if (!p.acc_init) ld256(p.acc + off, a1, a2);
                cmac(a1, p.acc_beta, L1);
                cmac(a2, p.acc_beta, L2);
                st256(p.acc + off, a1, a2);
            }
        }
        __syncwarp();
        if (AHEAD) failed = __any_sync(0xffffffffu, failed);
        unsigned char* const sw = slot;
        slot = slot_n;
        slot_n = sw;
        if (MI && ni != ci) {
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                hb_r[s] = nb_r[s];
                hb_i[s] = nb_i[s];
                ha_r[s] = na_r[s];
                ha_i[s] = na_i[s];
            }
            ci = ni;
        }
    }
    // a warp whose wait expired flags the launch as failed; before it leaves, the copies that no wait has seen arrive
    // (ADO it's, and the next one's where it was issued before that wait) get their time to land
    if (failed) {
        drain(bars + (it & 1), (it >> 1) & 1);
        if (!AHEAD && u + stride < nodes) drain(bars + ((it & 1) ^ 1), ((it + 1) >> 1) & 1);
        if (lane == 0) *static_cast<volatile int*>(dp.err) = 1;
    }
}

// ---------------------------------------------------------------------------
// Lockstep ensembles (N <= 8): K instances that share the hierarchy graph and
// the bath tables and differ in H only (the realisations of a static-disorder
// ensemble of one depth) are stored instance-minor: sector p of ADO u of
// instance k at sector index (u * P + p) * Kp + k (Kp = K rounded up to 32),
// so that the 32 instances of a block sit side by side in every row.
//
// Work item = (ADO u, block of 32 instances), swept grid-stride by a CTA of
// eight warps:
//   A  the block's 32 tiles arrive by 16-byte cp.async in a shared tile
//      [p][32] whose columns are swizzled (k ^ (p & 3)), which keeps the
//      conflict-free operand reads of the pair order; warp w computes the
//      commutator of instances w, w+8, w+16, w+24 on the tensor pipe (the
//      operand mapping of heom_dmma_stage); the result of a lane is that of
//      its own row elements and goes to a second shared tile, to the place
//      where the lane read them in the first;
//   B  warp w takes every eighth sector of a list whose first, ninth, ...
//      entries are the diagonal ones (half the terms: 7 states leave one warp
//      four of 25 sectors); lane k is instance k of the block.
//      Neighbour indices, tuple entries and bath coefficients are the same
//      for every lane (warp-uniform), and each neighbour read is one
//      contiguous 1-KB row (32 instances x 32 B) of the neighbour ADO, where
//      heom_dmma_stage gathers 32-B sectors of eight different neighbours.
// The derivative is the same element by element as heom_dmma_stage's (the
// same bath-term order; the commutator from the same MMA sequence).
// Instruction issue and the L1 data pipe bound it.  us per stage, one B200: 256
// instances of 7 states, depth 6: 245.3 -> 244.3 with the list and absent
// neighbours skipped (the terms of both sides now add up as heom_dmma_stage's
// do), -> 224.5 without an exchange of the commutator through shared memory, ->
// 219.8 with lanes outside the tile reading what one inside reads and sectors in an
// order searched for the reads that are made; 40 at depth 4: 18.8 -> 16.3 -> 14.4 ->
// 14.0; 256 of 6 states, depth 6: 107 -> 101 by the last step; 64 of 6 states, two
// slots, depth 4: 69.5 -> 68.7 -> 62.9 -> 57.4.
// ---------------------------------------------------------------------------

// ---------------------------------------------------------------------------
// N = 9..16: a team of TW warps per ADO, one thread per (state r, column pair
// t): thread r T + t of the team, T = ceil(N / 2), works as lane (r, t) of
// heom_dmma_stage does: it reads its two sectors {r, 2t}, {r, 2t+1} of the
// neighbours along the baths of state r, writes the sector it owns and hands
// the terms of the other one over to its owner.  The sectors are numbered in
// the order of their owners' threads.
//
// Commutator on the FP64 tensor pipe: the tile is zero-padded to 16 x 16 and
// cut into 2 x 2 blocks of 8 x 8; block (I, J) of C = w H - H w takes
// ceil(N/4) k-slices of m8n8k4 MMAs (A = w(8I+g, 4s+t) against the H
// fragment hb(J, s); ha(I, s) against B = w(4s+t, 8J+g)).  Warp wt of the
// team computes blocks [4 wt / TW, 4 (wt+1) / TW) and writes them to the
// team's exchange tile.
//
// Per ADO the team meets once: before the barrier every warp writes its blocks
// and its handed-over terms, and waits for its copies of the next ADO (two
// slots, cp.async); after it, the owners read the commutator and the terms
// handed to them, and the neighbours of the next ADO are asked for.  The
// exchange tile and the hand-over buffer alternate between two copies, so
// that no second barrier is needed.
//
// What bounds it: 18 to 20 warps per SM (96 registers) with the L1 data pipe
// 63 % busy (12 states, two slots: 514 wavefronts in 815 cycles per ADO and SM,
// 373 of them shared memory) and the FP64 tensor pipe a quarter.  Measured
// against a thread per sector with two barriers per ADO (us per stage, one
// B200): 12 states, two slots, 20,475 ADOs 74.5 -> 55.5 (24 warps of 80
// registers: 66) -> 53.4 with y read before the barrier, one slot, 18,564 ADOs
// 51.9 -> 43.1; 10 states, two slots, 10,626 ADOs 29.4 -> 24.4; 9 states, one
// slot, 5005 ADOs 13.9 -> 11.8; 11 states (three warps instead of two), one slot,
// 12,376 ADOs 29.3 -> 28.6; 16 states, two slots, 6545 ADOs 34.0 -> 27.3, one
// slot, 969 ADOs 8.21 -> 7.18, but 20,349 ADOs 75.2 -> 76.1 (with 106 registers
// and 16 warps 78.2).
// ---------------------------------------------------------------------------

// position of the sector owned by thread (r, t): threads of odd rows own
// nothing in the last column pair of an odd N
__host__ __device__ constexpr int team_pos(int n, int r, int t) { return r * ((n + 1) / 2) + t - ((n & 1) ? r >> 1 : 0); }

// CTAs per SM: 96 registers a thread where that does not spill (five warps on each SM partition), else 128 (four)
constexpr int team_blocks(int n, int hk, int slt)
{
    const bool small = hk == H_REAL_SYM && slt <= 2;
    return team_warps(n) == 3 ? (small ? 6 : 5) : (small ? 5 : 4);
}

// ADJ: the adjoint operator L^H (see heom_dmma_stage, also for K and C).  The
// bath coefficients are the factored tables of heom_dmma_stage (CoefTabs).
template <int N, int HK, int SLT, bool ADJ>
__global__ void __launch_bounds__(team_threads(N), team_blocks(N, HK, SLT))
    heom_pair_stage(const __grid_constant__ DmmaParams dp)
{
    static_assert(N > 8 && N <= 16, "team kernel handles N = 9..16");
    constexpr int P = pairs_of(N);
    constexpr int T = (N + 1) / 2;
    constexpr int TW = team_warps(N);
    constexpr int TT = 32 * TW;
    constexpr int KS = (N + 3) / 4; // k-slices of the padded commutator
    constexpr int FD = frag_doubles(N);
    constexpr int QB = SLT < 2 ? SLT : 2; // slots whose neighbours are read in one batch
    constexpr bool ODD = (N & 1) != 0;
    extern __shared__ __align__(128) unsigned char smem[];
    const PairParams& p = dp.p;
    const PairSmem L = pair_smem_layout(N, p.W, p.NW, p.TWB, p.LS);
    const int W = p.W, LS = p.LS, SL = p.SL;

    grid_launch_dependents();
    double2* s_kh = reinterpret_cast<double2*>(smem);      // [3][W]: kappa_i, kappa_j, kappa_i + kappa_j
    double2* s_sq = s_kh + 3 * W;                           // LS + 1: (sqrt(n), sqrt(n+1))
    double* s_ch = reinterpret_cast<double*>(s_sq + LS + 1); // W
    for (int q = threadIdx.x; q < 3 * W; q += blockDim.x) s_kh[q] = dp.ct.khat[q];
    for (int q = threadIdx.x; q < W; q += blockDim.x) s_ch[q] = dp.ct.chat[q];
    for (int q = threadIdx.x; q <= LS; q += blockDim.x)
        s_sq[q] = make_double2(dp.ct.sq[q], q < LS ? dp.ct.sq[q + 1] : 0.0);

    const int team = threadIdx.x / TT;
    const int lt = threadIdx.x - team * TT;
    unsigned char* team_base = smem + L.lut + team * L.team;
    const int wt = lt >> 5, lane = lt & 31, g = lane >> 2, t4 = lane & 3;
    const int blk0 = wt * 4 / TW, blk1 = (wt + 1) * 4 / TW; // commutator blocks of this warp
    // operand and result positions of block (0, 0) and slice 0 (tile_pos: the swap of columns k ^ (i & 2) leaves
    // multiples of four alone, so that blocks and slices add constants)
    constexpr int TS = tile_stride(N);
    const int oa = g * TS + (t4 ^ (g & 2)), ob = t4 * TS + (g ^ (t4 & 2)), xw = g * kXchStride + 2 * t4;

    // ---- this thread's place ----
    const bool active = lt < N * T;
    const int r = active ? lt / T : 0, t = active ? lt - r * T : 0, R = r >> 1;
    const int odd = row_owned(r, t);                        // owns {r, 2t + odd}
    const int co = 2 * t + odd, cg = 2 * t + 1 - odd;       // columns owned, handed over
    const bool dga = t == R && !(r & 1), dgb = t == R && (r & 1); // the diagonal sector is owned / handed over
    const bool owner = active && co < N, holds = active && cg < N;
    const int ro = t == R ? r ^ 1 : cg, tr = t == R ? t : R; // row and column pair of the thread that owns it
    const int pso = team_pos(N, r, t), psg = team_pos(N, ro, tr), rid = ro * T + tr;
    const int i2 = dga ? (r + 1 < N ? r + 1 : r) : co, j2 = dga ? i2 : r; // second element of the owned sector
    const int tp1 = owner ? tile_pos(N, r, co) : 0, tp2 = owner ? tile_pos(N, i2, j2) : 0;
    const int xc1 = r * kXchStride + co, xc2 = i2 * kXchStride + j2;
    // negative: no such sector; no C term on it (diagonal)
    const int no_o = owner ? 0 : -1, no_g = holds ? 0 : -1;
    const int no_co = dga ? -1 : no_o, no_cg = dgb ? -1 : no_g;
    const double2* in_o = p.in + 2 * (owner ? pso : 0);
    const double2* in_g = p.in + 2 * (holds ? psg : 0);

    int slo[SLT], kp[SLT]; // slots of state r and their table positions (-1: none)
#pragma unroll
    for (int q = 0; q < SLT; ++q) {
        const int sl = (active && q < SL) ? p.slots[r * SL + q] : -1;
        slo[q] = sl >= 0 ? sl : 0;
        kp[q] = sl >= 0 ? dp.ct.pos[sl] : -1;
    }
    const double2* kt_of = s_kh + (dga ? 2 : 0) * W;
    const double2* kt_gs = s_kh + (dgb ? 2 : 0) * W;
    const double2* kt_j = s_kh + W;
    double2* s_gam = reinterpret_cast<double2*>(team_base + L.gam_off); // [2][TT]: gamma0 of the owned elements
    s_gam[lt] = owner ? p.gamma0[r * N + co] : make_double2(0.0, 0.0);
    s_gam[TT + lt] = owner ? p.gamma0[i2 * N + j2] : make_double2(0.0, 0.0);
    // terms handed over, two copies of [2][TT]; what nobody hands over (the last diagonal element of an odd N) stays zero
    double2* hand = reinterpret_cast<double2*>(team_base + L.hand_off);
    for (int q = 0; q < 4; ++q) hand[q * TT + lt] = make_double2(0.0, 0.0);
    __syncthreads();

    const unsigned nodes = (unsigned)p.nodes; // at most 2^31 - 1
    constexpr int TEAMS = cta_teams(N);
    const unsigned stride = gridDim.x * TEAMS;
    unsigned u = blockIdx.x * TEAMS + team;
    const int recb = rec_bytes(p.NW, p.TWB);

    // issue the asynchronous copies of ADO v into a slot: its own sector by every owner (scattered into the
    // row-major tile), the record by the first threads
    auto prefetch = [&](unsigned v, unsigned char* slot) {
        double2* tile = reinterpret_cast<double2*>(slot + L.tile_off);
        if (owner) {
            const double2* src = in_o + (int64_t)v * (2 * P);
            cp_async16(tile + tp1, src);
            cp_async16(tile + tp2, src + 1);
        }
        for (int q = lt * 16; q < recb; q += TT * 16) cp_async16(slot + L.nbr_off + q, p.rec + (int64_t)v * recb + q);
    };
    // the neighbours of the first slots' batch (QB slots) are read one ADO ahead: vk, vc their indices along K and C,
    // xo, xg the K neighbours' sectors
    int vk[QB], vc[QB];
    double2 xo[QB][2], xg[QB][2];
    auto index = [&](const unsigned char* rec, int q0) {
        const int2* nb = reinterpret_cast<const int2*>(rec);
#pragma unroll
        for (int b = 0; b < QB; ++b) {
            const int2 pm = kp[q0 + b] >= 0 ? nb[slo[q0 + b]] : make_int2(-1, -1);
            vk[b] = ADJ ? pm.x : pm.y;
            vc[b] = ADJ ? pm.y : pm.x;
        }
    };
    auto load_k = [&]() {
#pragma unroll
        for (int b = 0; b < QB; ++b) {
            const int64_t o = (int64_t)vk[b] * (2 * P);
            ld256_if(ODD ? vk[b] | no_o : vk[b], in_o + o, xo[b][0], xo[b][1]);
            ld256_if(ODD ? vk[b] | no_g : vk[b], in_g + o, xg[b][0], xg[b][1]);
        }
    };

    // the first ADO's indices come from the record array, so that its neighbours are asked for together with its tile
    if (u < nodes) index(p.rec + (int64_t)u * recb, 0);
    grid_wait(); // the state and the H tables of a field are written by the kernels before this one
    unsigned it = 0;
    if (u < nodes) {
        prefetch(u, team_base);
        load_k();
    }
    cp_async_wait_all();
    team_sync<TW>(team);
    for (; u < nodes; u += stride, ++it) {
        const unsigned char* slot = team_base + (it & 1) * L.slot;
        unsigned char* slot_n = team_base + ((it & 1) ^ 1) * L.slot;
        const bool more = u + stride < nodes;
        if (more) prefetch(u + stride, slot_n); // its last readers are behind the barrier of the previous iteration
        const double2* tile = reinterpret_cast<const double2*>(slot + L.tile_off);
        const unsigned char* tu = slot + L.tup_off;
        double2* xch = reinterpret_cast<double2*>(team_base + L.xch_off + (it & 1) * kXchBytes);
        double2* hnd = hand + (it & 1) * 2 * TT;

        // ---- commutator w H - H w / hbar on the tensor pipe, into the exchange tile ----
        // (rows and columns of an operand outside N x N are not read from the result and may hold anything; a
        // contraction index outside must be zero)
        const double* fr = p.hfrag + (p.inst ? (size_t)__ldg(p.inst + u) * FD : 0) + lane;
        const double2* ta = tile + oa;
        const double2* tb = tile + ob;
#pragma unroll
        for (int blk = 0; blk < 4; ++blk) {
            if (blk < blk0 || blk >= blk1) continue;
            const int I = blk >> 1, J = blk & 1;
            double cr0 = 0.0, cr1 = 0.0, ci0 = 0.0, ci1 = 0.0;
#pragma unroll
            for (int s = 0; s < KS; ++s) {
                // A = w(8I+g, 4s+t4), B = w(4s+t4, 8J+g)
                const bool in = 4 * s + 3 < N || 4 * s + t4 < N;
                const double2 z = make_double2(0.0, 0.0);
                const double2 A = in ? ta[8 * I * TS + 4 * s] : z;
                const double2 B = in ? tb[8 * J + 4 * s * TS] : z;
                const double hbr = fr[frag_index(N, 0, J, s, 0)];
                dmma(cr0, cr1, A.x, hbr); // Re(w) Re(H)
                dmma(ci0, ci1, A.y, hbr); // Im(w) Re(H)
                if (HK == H_GENERIC) {
                    const double har = fr[frag_index(N, 2, I, s, 0)];
                    const double hbi = fr[frag_index(N, 1, J, s, 0)];
                    const double hai = fr[frag_index(N, 3, I, s, 0)];
                    dmma(cr0, cr1, har, B.x);  // -Re(H) Re(w)
                    dmma(ci0, ci1, har, B.y);  // -Re(H) Im(w)
                    dmma(cr0, cr1, -A.y, hbi); // -Im(w) Im(H)
                    dmma(ci0, ci1, A.x, hbi);  //  Re(w) Im(H)
                    dmma(cr0, cr1, -hai, B.y); // +Im(H) Im(w)
                    dmma(ci0, ci1, hai, B.x);  // -Im(H) Re(w)
                } else { // H(r, k) = H(k, r): block I's fragment of w H is that of H w with the sign changed
                    const double hir = I == J ? hbr : fr[frag_index(N, 0, I, s, 0)];
                    dmma(cr0, cr1, hir, -B.x);
                    dmma(ci0, ci1, hir, -B.y);
                }
            }
            double2* xr = xch + xw + 8 * I * kXchStride + 8 * J;
            xr[0] = make_double2(cr0, ci0);
            xr[1] = make_double2(cr1, ci1);
        }

        // ---- same term of the owned elements ----
        double2 pss = *reinterpret_cast<const double2*>(slot + L.pss_off);
        if (p.no_same) pss = make_double2(0.0, 0.0);
        if (ADJ) pss.y = -pss.y;
        const double2 xf = tile[tp1], xs = tile[tp2];
        double2 of = make_double2(0.0, 0.0), os = of, gf = of, gs = of; // owned / handed-over sector, first / second half
        {
            const double2 g1 = s_gam[lt], g2 = s_gam[TT + lt];
            cmac(of, make_double2(pss.x + g1.x, pss.y + g1.y), xf);
            cmac(os, make_double2(pss.x + g2.x, pss.y + g2.y), xs);
        }
        // what the stage adds to: y takes the place of the own values, in flight through the bath terms (a launch with
        // y never starts acc from the own values)
        double2 x1 = xf, x2 = xs;
        if (p.y && owner) ld256(p.y + (int64_t)u * (2 * P) + 2 * pso, x1, x2);
#pragma unroll
        for (int q0 = 0; q0 < SLT; q0 += QB) {
            if (q0 > 0) {
                index(slot + L.nbr_off, q0);
                load_k();
            }
            // ---- bath terms: K neighbours ----
#pragma unroll
            for (int b = 0; b < QB; ++b) {
                const int q = q0 + b;
                if (vk[b] >= 0) {
                    const double2* sq = s_sq + tu[slo[q]];
                    const double sk = ADJ ? sq->y : sq->x;
                    auto kap = [&](const double2* tab) {
                        const double2 v = tab[kp[q]];
                        return make_double2(v.x * sk, (ADJ ? -v.y : v.y) * sk);
                    };
                    cmac(of, kap(kt_of), xo[b][0]);
                    cmac(gs, kap(kt_gs), xg[b][1]);
                    const double2 k = kap(kt_j);
                    if (!dga) cmac(os, k, xo[b][1]);
                    if (!dgb) cmac(gf, k, xg[b][0]);
                }
            }
            // ---- C neighbours (a diagonal element's terms of its row and column cancel) ----
#pragma unroll
            for (int b = 0; b < QB; ++b) {
                const int64_t o = (int64_t)vc[b] * (2 * P);
                if (vc[b] >= 0) {
                    ld256_if(no_co, in_o + o, xo[b][0], xo[b][1]);
                    ld256_if(no_cg, in_g + o, xg[b][0], xg[b][1]);
                }
            }
#pragma unroll
            for (int b = 0; b < QB; ++b) {
                const int q = q0 + b;
                if (vc[b] >= 0) {
                    const double2 sq = s_sq[tu[slo[q]]];
                    const double c = ADJ ? -s_ch[kp[q]] * sq.x : s_ch[kp[q]] * sq.y;
                    if (!dga) {
                        of.x = fma(-c, xo[b][0].y, of.x);
                        of.y = fma(c, xo[b][0].x, of.y);
                        os.x = fma(c, xo[b][1].y, os.x);
                        os.y = fma(-c, xo[b][1].x, os.y);
                    }
                    if (!dgb) {
                        gf.x = fma(c, xg[b][0].y, gf.x);
                        gf.y = fma(-c, xg[b][0].x, gf.y);
                        gs.x = fma(-c, xg[b][1].y, gs.x);
                        gs.y = fma(c, xg[b][1].x, gs.y);
                    }
                }
            }
        }
        if (holds) {
            hnd[rid] = gf;
            hnd[TT + rid] = gs;
        }
        cp_async_wait_all();
        team_sync<TW>(team);
        if (more) { // in flight through the stores and the next commutator
            index(slot_n + L.nbr_off, 0);
            load_k();
        }

        if (owner) {
            // ---- commutator i * (w H - H w) / hbar and the terms handed over ----
            const double2 c1 = xch[xc1], c2 = xch[xc2], hf = hnd[lt], hs = hnd[TT + lt];
            const double2 L1 = make_double2((of.x - c1.y) + hf.x, (of.y + c1.x) + hf.y);
            double2 L2 = make_double2((os.x - c2.y) + hs.x, (os.y + c2.x) + hs.y);
            if (ODD && dga && r == N - 1) L2 = L1; // the padding half mirrors its element

            // ---- stage write ----
            const int64_t off = (int64_t)u * (2 * P) + 2 * pso;
            double2 r1 = p.use_x ? x1 : make_double2(0.0, 0.0), r2 = p.use_x ? x2 : make_double2(0.0, 0.0);
            cmac(r1, p.beta, L1);
            cmac(r2, p.beta, L2);
            st256_cs(p.out + off, r1, r2);
            if (p.use_acc) {
                double2 a1 = x1, a2 = x2;
                if (!p.acc_init) ld256(p.acc + off, a1, a2);
                cmac(a1, p.acc_beta, L1);
                cmac(a2, p.acc_beta, L2);
                st256(p.acc + off, a1, a2);
            }
        }
    }
}

// out = y + h * sum_l c_l k_l over doubles, terms with c_l == 0 skipped, in
// the operation order of rk_weighted_add.cl:78-95 (no contraction).
struct WaddParams {
    double* out;
    const double* y;
    const double* k[7];
    double c[7];
    int n;
    double h;
    int64_t len;
};

__global__ void heom_weighted_add(const WaddParams p)
{
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < p.len; e += stride) {
        double acc = 0.0;
        for (int l = 0; l < p.n; ++l)
            if (p.c[l] != 0.0) acc = __dadd_rn(acc, __dmul_rn(p.c[l], p.k[l][e]));
        acc = __dmul_rn(acc, p.h);
        acc = __dadd_rn(acc, p.y[e]);
        p.out[e] = acc;
    }
}

// Reference layout (row-major tiles in uid order) <-> pair layout in the
// internal ADO order, over the reference ADOs [r0, r0 + count) whose tiles
// are (or go) back to back in `ref`.  pe[2p], pe[2p+1] = element indices of
// the halves of sector p (equal for the padding half).  One thread per
// (ADO, sector): the pair side is written / read as whole 32-byte sectors.
__global__ void heom_to_pairs(double2* __restrict__ dst, const double2* __restrict__ ref,
                              const int64_t* __restrict__ int_of_ref, const int16_t* __restrict__ pe,
                              int64_t r0, int64_t count, int n, int P)
{
    const int64_t total = count * P;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += stride) {
        const int64_t r = q / P;
        const int pr = (int)(q - r * P);
        const int64_t u = int_of_ref[r0 + r];
        const double2* src = ref + r * n * n;
        dst[(u * P + pr) * 2] = src[pe[2 * pr]];
        dst[(u * P + pr) * 2 + 1] = src[pe[2 * pr + 1]];
    }
}

__global__ void heom_from_pairs(double2* __restrict__ ref, const double2* __restrict__ src,
                                const int64_t* __restrict__ int_of_ref, const int16_t* __restrict__ pe,
                                int64_t r0, int64_t count, int n, int P)
{
    const int64_t total = count * P;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += stride) {
        const int64_t r = q / P;
        const int pr = (int)(q - r * P);
        const int64_t u = int_of_ref[r0 + r];
        double2* dst = ref + r * n * n;
        const int e1 = pe[2 * pr], e2 = pe[2 * pr + 1];
        dst[e1] = src[(u * P + pr) * 2];
        if (e2 != e1) dst[e2] = src[(u * P + pr) * 2 + 1];
    }
}

// Copy the top matrix of every instance (block k: internal ADO tops[k], pair
// layout) into row `row` of a row-major log [rows][n_inst][n*n].
// sector index of sector p of internal ADO u: the per-instance layout (kp = 0)
// or the lockstep layout of instance k (stride kp)
__device__ __forceinline__ int64_t sector_index(int64_t u, int p, int P, int64_t kp, int64_t k)
{
    return kp ? (u * P + p) * kp + k : u * P + p;
}

// block b: the instance k0 + b of a lockstep handle (kp > 0), ignored otherwise
__global__ void heom_record_top(double2* __restrict__ log, const double2* __restrict__ y,
                                const int16_t* __restrict__ pe, const int64_t* __restrict__ tops, int n, int P,
                                int64_t row, int64_t kp, int64_t k0)
{
    const int k = blockIdx.x;
    const int64_t u = tops[k];
    double2* dst = log + (row * gridDim.x + k) * n * n;
    for (int pr = threadIdx.x; pr < P; pr += blockDim.x) {
        const int e1 = pe[2 * pr], e2 = pe[2 * pr + 1];
        const int64_t sx = sector_index(u, pr, P, kp, k0 + k);
        dst[e1] = y[sx * 2];
        if (e2 != e1) dst[e2] = y[sx * 2 + 1];
    }
}

// heom_record_top into row *base + j (a device offset, for captured graphs)
__global__ void heom_record_top_at(double2* __restrict__ log, const double2* __restrict__ y,
                                   const int16_t* __restrict__ pe, const int64_t* __restrict__ tops, int n, int P,
                                   const int64_t* __restrict__ base, int64_t j)
{
    const int k = blockIdx.x;
    const int64_t u = tops[k];
    double2* dst = log + ((*base + j) * gridDim.x + k) * n * n;
    for (int pr = threadIdx.x; pr < P; pr += blockDim.x) {
        const int e1 = pe[2 * pr], e2 = pe[2 * pr + 1];
        dst[e1] = y[(u * P + pr) * 2];
        if (e2 != e1) dst[e2] = y[(u * P + pr) * 2 + 1];
    }
}

// Write row-major top matrices top[k] ([n_inst][n*n]) into the pair layout
// of each instance's top ADO (block k).
__global__ void heom_write_top(double2* __restrict__ y, const double2* __restrict__ top,
                               const int16_t* __restrict__ pe, const int64_t* __restrict__ tops, int n, int P,
                               int64_t kp, int64_t k0)
{
    const int k = blockIdx.x;
    const int64_t u = tops[k];
    const double2* src = top + (int64_t)k * n * n;
    for (int pr = threadIdx.x; pr < P; pr += blockDim.x) {
        const int64_t sx = sector_index(u, pr, P, kp, k0 + k);
        y[sx * 2] = src[pe[2 * pr]];
        y[sx * 2 + 1] = src[pe[2 * pr + 1]];
    }
}

// ---------------------------------------------------------------------------
// Adjoint gradients.  For one RK4 stage factor F_k = I + beta_k h L of the
// product form, dJ/dtheta gains Re(beta_k h <a, dL/dtheta w>), with a the
// adjoint after the later factors and w the stage input (<x, y> = x^H y).
//   H:      <a, dL/dH_ab w> = (i/hbar) Z(a,b),
//           Z = sum_u (w_u^T conj(a_u) - conj(a_u) w_u^T)          (all a, b at once)
//   lambda, gamma (shared by all baths): L is linear in its coefficient
//           tables, so dL/dtheta is L with H = 0 and the tables replaced by
//           their derivatives (dpss, dgamma0, dchat, dkhat).
// One warp per ADO; its lanes take the (state, column pair) threads of the
// stage kernels in turn, so that the look-ups of a slot serve four elements, and
// the derivative tables lie in shared memory.  Latency bounds it, so that two
// blocks on an SM count for more than the 32 bytes that 128 registers spill, and
// a warp's sums lie where its tiles were (16 states: 86 KB a block).  Whole
// gradient calls, one B200, with one block of 158 registers -> with two: 4
// instances of 9 states, 715 ADOs each, 40 steps 7220 -> 6910 us; 12 states, two
// slots, 20,475 ADOs, 8 steps 10,840 -> 9150; 16 states, 4845 ADOs, 20 steps
// 10,900 -> 9540 (a lane per sector, tables in global memory, two blocks of 126
// registers: 8410, 12,200 and 9990).  The blocks are split
// among the instances of the handle (each block sweeps one instance's ADOs),
// and every block adds weight * (its sum) to its own row of `partial`
// (deterministic; summed per instance on the host at the end).
// ---------------------------------------------------------------------------
struct GradParams {
    const double2* __restrict__ a;     // adjoint (pair layout, internal order)
    const double2* __restrict__ w;     // forward stage input
    const unsigned char* __restrict__ rec; // [nodes] records: (plus, minus) of every slot, tuple bytes
    const int16_t* __restrict__ pe;    // [2P] element indices of the sector halves
    const int16_t* __restrict__ slots; // [N][SL] slot ids of each state, -1 padded
    const double* __restrict__ dpss;   // [nodes] d pf_same_sum / d gamma (real)
    const double2* __restrict__ dg0;   // [2][N*N] d gamma0 / d(lambda, gamma)
    const double* __restrict__ dchat;  // [2][W] d chat
    const double2* __restrict__ dkhat; // [2][3][W] d khat (side i, side j, diagonal)
    const double* __restrict__ sq;     // [LS+1] sqrt(n)
    // one launch takes `factors` pairs (a, w) that follow one another in the backward sweep: pair f at a + f a_step,
    // w + f w_step (double2 elements), its weight beta_k h with k = factor0 - f (mod 4)
    int factors, factor0;
    int64_t a_step, w_step;
    double2 weight[4];
    RowTab rt;                         // heom_row_grad
    double2* partial;                  // [gridDim.x][N*N + 2]
    const int64_t* inst_base;          // [instances + 1] first ADO of every instance
    int blocks_per_inst;               // blocks [k*bpi, (k+1)*bpi) sweep instance k only
    int N, P, W, NW, TWB, SL, LS;
    int want_h;                        // accumulate Z (the H gradient)
    int want_bath;                     // accumulate <a, L_theta' w> (the lambda and gamma gradients)
};

// one (state, column pair) of heom_adjoint_grad, as a lane of the stage kernels: its owned and handed-over sector
// (-1: none), the elements of the owned one, tile positions of its halves and of the other's row and column element
struct GradLane {
    short r, diag, pso, psg, e1, e2, q1, q2, gr, gc, twin, pad; // diag 1: the owned sector is diagonal, 2: the other
};
// a warp's two tiles [n][n+1]; at the end of a factor its n*n + 2 sums lie there
__host__ __device__ constexpr int grad_warp_bytes(int n) { return 2 * n * (n + 1) * 16; }
__host__ inline size_t grad_smem_bytes(int n, int W, int LS)
{
    return (size_t)kCtaWarps * grad_warp_bytes(n) + (size_t)(n * n + 2) * 16 +
           (size_t)(2 * n * n + 5 * W) * 16 + (size_t)((LS + 2) & ~1) * 8 + (size_t)n * ((n + 1) / 2) * sizeof(GradLane);
}

__global__ void __launch_bounds__(kCtaWarps * 32, 2) heom_adjoint_grad(const __grid_constant__ GradParams g)
{
    extern __shared__ __align__(128) unsigned char smem[];
    const int N = g.N, P = g.P, W = g.W, SL = g.SL, NN = N * N, LD = N + 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double2* At = reinterpret_cast<double2*>(smem + warp * grad_warp_bytes(N)); // [N][N+1]
    double2* Wt = At + N * LD;
    double2* acc = reinterpret_cast<double2*>(smem + kCtaWarps * grad_warp_bytes(N)); // [NN+2]
    // derivative tables, lambda and gamma side by side: dg0 [NN][2], dkhat side i and side j [W][4], dchat [W]
    double2* s_dg = acc + NN + 2;
    double2* s_dk = s_dg + 2 * NN;
    double2* s_dc = s_dk + 4 * W;
    double* s_sq = reinterpret_cast<double*>(s_dc + W);                                // [LS+1]
    GradLane* lanes = reinterpret_cast<GradLane*>(s_sq + ((g.LS + 2) & ~1));           // [N T]
    for (int q = threadIdx.x; q < 2 * NN; q += blockDim.x) s_dg[q] = g.dg0[(q & 1) * NN + (q >> 1)];
    for (int q = threadIdx.x; q < 4 * W; q += blockDim.x) s_dk[q] = g.dkhat[(q & 1) * 3 * W + ((q >> 1) & 1) * W + (q >> 2)];
    for (int q = threadIdx.x; q < W; q += blockDim.x) s_dc[q] = make_double2(g.dchat[q], g.dchat[W + q]);
    for (int q = threadIdx.x; q <= g.LS; q += blockDim.x) s_sq[q] = g.sq[q];
    const int T = (N + 1) / 2, NL = N * T;
    for (int l = threadIdx.x; l < NL; l += blockDim.x) {
        const int r = l / T, t = l - r * T, R = r >> 1, odd = row_owned(r, t);
        const int co = 2 * t + odd, cg = 2 * t + 1 - odd;
        const bool dga = t == R && !(r & 1), dgb = t == R && (r & 1);
        GradLane q;
        q.r = r;
        q.diag = dga ? 1 : dgb ? 2 : 0;
        q.pso = q.psg = -1;
        for (int p = 0; p < P; ++p) { // the sectors that hold (r, co) and (r, cg)
            const int e1 = g.pe[2 * p], e2 = g.pe[2 * p + 1];
            if (co < N && (e1 == r * N + co || e2 == r * N + co)) q.pso = p;
            if (cg < N && (e1 == r * N + cg || e2 == r * N + cg)) q.psg = p;
        }
        const int i2 = dga ? (r + 1 < N ? r + 1 : r) : co, j2 = dga ? i2 : r;
        q.twin = dga && i2 == r;
        q.e1 = co < N ? r * N + co : 0;
        q.e2 = co < N ? i2 * N + j2 : 0;
        q.q1 = co < N ? r * LD + co : 0;
        q.q2 = co < N ? i2 * LD + j2 : 0;
        q.gr = cg < N ? r * LD + cg : 0;
        q.gc = cg < N ? (dgb ? q.gr : cg * LD + r) : 0;
        lanes[l] = q;
    }
    // Z on the FP64 tensor pipe: blocks (I, J) of 8 x 8 of the zero-padded Z (one block for
    // N <= 8, 2 x 2 for N <= 16), accumulated over the warp's ADOs in the MMA fragments:
    // lane 4g + t holds Z(8I+g, 8J+2t) and Z(8I+g, 8J+2t+1), real and imaginary parts
    const int gq = lane >> 2, t4 = lane & 3;
    const int nblk = N <= 8 ? 1 : 4, ks = (N + 3) / 4;
    double zr[4][2], zi[4][2];
    auto el = [&](const double2* T, int r, int c) {
        return (r < N && c < N) ? T[r * LD + c] : make_double2(0.0, 0.0);
    };
    auto conj_mac = [](double2& s, const double2 a, const double2 w) { // s += conj(a) w
        s.x = fma(a.x, w.x, s.x);
        s.x = fma(a.y, w.y, s.x);
        s.y = fma(a.x, w.y, s.y);
        s.y = fma(-a.y, w.x, s.y);
    };

    const int inst = blockIdx.x / g.blocks_per_inst, jb = blockIdx.x - inst * g.blocks_per_inst;
    const int64_t stride = (int64_t)g.blocks_per_inst * kCtaWarps, end = g.inst_base[inst + 1];
    double2* const out = g.partial + (int64_t)blockIdx.x * (NN + 2);
    for (int q = threadIdx.x; q < NN + 2; q += blockDim.x) acc[q] = out[q];
    __syncthreads();
    for (int f = 0; f < g.factors; ++f) {
        const double2* a_in = g.a + f * g.a_step;
        const double2* w_in = g.w + f * g.w_step;
        const double2 z0 = make_double2(0.0, 0.0);
#pragma unroll
        for (int b = 0; b < 4; ++b) zr[b][0] = zr[b][1] = zi[b][0] = zi[b][1] = 0.0;
        double2 dl = z0, dgm = z0;
        for (int64_t u = g.inst_base[inst] + (int64_t)jb * kCtaWarps + warp; u < end; u += stride) {
            const unsigned char* nb = g.rec + u * rec_bytes(g.NW, g.TWB);
            const unsigned char* tu = nb + g.NW * 4;
            const double dps = g.dpss[u];
            for (int l = lane; l < NL; l += 32) {
                const GradLane q = lanes[l];
                if (q.pso < 0) continue;
                double2 a1, a2, w1, w2;
                ld256(a_in + (u * P + q.pso) * 2, a1, a2);
                ld256(w_in + (u * P + q.pso) * 2, w1, w2);
                At[q.q1] = a1;
                At[q.q2] = a2;
                Wt[q.q1] = w1;
                Wt[q.q2] = w2;
            }
            __syncwarp();
            if (g.want_bath)
                for (int l = lane; l < NL; l += 32) {
                    const GradLane q = lanes[l];
                    const double2 a1 = At[q.q1], a2 = At[q.q2], ar = At[q.gr], ac = At[q.gc];
                    // same term of the owned elements (a padding half counts once)
                    if (q.pso >= 0) {
                        double2 v1 = z0, v2 = z0;
                        conj_mac(v1, a1, Wt[q.q1]);
                        if (!q.twin) conj_mac(v2, a2, Wt[q.q2]);
                        cmac(dl, s_dg[2 * q.e1], v1);
                        cmac(dl, s_dg[2 * q.e2], v2);
                        const double2 s1 = s_dg[2 * q.e1 + 1], s2 = s_dg[2 * q.e2 + 1];
                        cmac(dgm, make_double2(s1.x + dps, s1.y), v1);
                        cmac(dgm, make_double2(s2.x + dps, s2.y), v2);
                    }
                    for (int k = 0; k < SL; ++k) {
                        const int sl = g.slots[q.r * SL + k];
                        if (sl < 0) continue;
                        const int2 pm = __ldg(reinterpret_cast<const int2*>(nb) + sl);
                        const int n = tu[sl];
                        double2 mo[2], mg[2], po[2], pg[2]; // minus and plus neighbour, owned and handed-over sector
                        const int no = q.pso < 0 ? -1 : 0, ng = q.psg < 0 ? -1 : 0;
                        const int co = q.diag == 1 ? -1 : no, cg = q.diag == 2 ? -1 : ng; // plus terms of a diagonal cancel
                        const double2* bo = w_in + (q.pso < 0 ? 0 : q.pso) * 2;
                        const double2* bg = w_in + (q.psg < 0 ? 0 : q.psg) * 2;
                        ld256_if(pm.y | no, bo + (int64_t)pm.y * (2 * P), mo[0], mo[1]);
                        ld256_if(pm.y | ng, bg + (int64_t)pm.y * (2 * P), mg[0], mg[1]);
                        ld256_if(pm.x | co, bo + (int64_t)pm.x * (2 * P), po[0], po[1]);
                        ld256_if(pm.x | cg, bg + (int64_t)pm.x * (2 * P), pg[0], pg[1]);
                        if (pm.y >= 0) {
                            double2 vi = z0, vj = z0; // row and column elements
                            if (no >= 0) {
                                conj_mac(vi, a1, mo[0]);
                                conj_mac(vj, q.diag == 1 ? a1 : a2, q.diag == 1 ? mo[0] : mo[1]);
                            }
                            if (ng >= 0) {
                                conj_mac(vi, ar, mg[1]);
                                conj_mac(vj, ac, q.diag == 2 ? mg[1] : mg[0]);
                            }
                            const double s = s_sq[n];
                            vi = make_double2(vi.x * s, vi.y * s);
                            vj = make_double2(vj.x * s, vj.y * s);
                            const double2* dk = s_dk + 4 * sl;
                            cmac(dl, dk[0], vi);
                            cmac(dgm, dk[1], vi);
                            cmac(dl, dk[2], vj);
                            cmac(dgm, dk[3], vj);
                        }
                        if (pm.x >= 0) {
                            double2 vr = z0, vc = z0; // row elements with +i, column elements with -i
                            if (co >= 0) {
                                conj_mac(vr, a1, po[0]);
                                conj_mac(vc, a2, po[1]);
                            }
                            if (cg >= 0) {
                                conj_mac(vr, ar, pg[1]);
                                conj_mac(vc, ac, pg[0]);
                            }
                            const double s = s_sq[n + 1];
                            const double vx = s * (vc.y - vr.y), vy = s * (vr.x - vc.x); // i (vr - vc)
                            const double2 c = s_dc[sl];
                            dl.x = fma(c.x, vx, dl.x);
                            dl.y = fma(c.x, vy, dl.y);
                            dgm.x = fma(c.y, vx, dgm.x);
                            dgm.y = fma(c.y, vy, dgm.y);
                        }
                    }
                }
            // Z(k,l) = sum_i w(i,k) conj(a(i,l)) - sum_j conj(a(k,j)) w(l,j):
            //   Re Z = Wr^T Ar + Wi^T Ai - Ar Wr^T - Ai Wi^T, Im Z = Wi^T Ar - Wr^T Ai - Ar Wi^T + Ai Wr^T
            if (g.want_h) {
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    if (b >= nblk) continue;
                    const int I = b >> 1, J = b & 1;
#pragma unroll
                    for (int s = 0; s < 4; ++s) {
                        if (s >= ks) continue;
                        const int k0 = 4 * s + t4;
                        const double2 wT = el(Wt, k0, 8 * I + gq); // A operand of W^T A: W(4s+t, 8I+g)
                        const double2 aB = el(At, k0, 8 * J + gq); // B operand of W^T A: A(4s+t, 8J+g)
                        const double2 aA = el(At, 8 * I + gq, k0); // A operand of A W^T: A(8I+g, 4s+t)
                        const double2 wB = el(Wt, 8 * J + gq, k0); // B operand of A W^T: W(8J+g, 4s+t)
                        dmma(zr[b][0], zr[b][1], wT.x, aB.x);
                        dmma(zr[b][0], zr[b][1], wT.y, aB.y);
                        dmma(zr[b][0], zr[b][1], -aA.x, wB.x);
                        dmma(zr[b][0], zr[b][1], -aA.y, wB.y);
                        dmma(zi[b][0], zi[b][1], wT.y, aB.x);
                        dmma(zi[b][0], zi[b][1], -wT.x, aB.y);
                        dmma(zi[b][0], zi[b][1], -aA.x, wB.y);
                        dmma(zi[b][0], zi[b][1], aA.y, wB.x);
                    }
                }
            }
            __syncwarp();
        }
        // block sum in a fixed order, then weight * sum into this block's row
        double2* mine = At; // [NN+2], where the warp's tiles were
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            if (b >= nblk) continue;
            const int r = 8 * (b >> 1) + gq;
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int c = 8 * (b & 1) + 2 * t4 + e;
                if (r < N && c < N) mine[r * N + c] = make_double2(zr[b][e], zi[b][e]);
            }
        }
        for (int off = 16; off > 0; off >>= 1) {
            dl.x += __shfl_down_sync(0xffffffffu, dl.x, off);
            dl.y += __shfl_down_sync(0xffffffffu, dl.y, off);
            dgm.x += __shfl_down_sync(0xffffffffu, dgm.x, off);
            dgm.y += __shfl_down_sync(0xffffffffu, dgm.y, off);
        }
        if (lane == 0) {
            mine[NN] = dl;
            mine[NN + 1] = dgm;
        }
        __syncthreads();
        const double2 wgt = g.weight[(g.factor0 - f) & 3];
        for (int q = threadIdx.x; q < NN + 2; q += blockDim.x) {
            double2 s = z0;
            for (int v = 0; v < kCtaWarps; ++v) {
                const double2 m = reinterpret_cast<const double2*>(smem + v * grad_warp_bytes(N))[q];
                s.x += m.x;
                s.y += m.y;
            }
            acc[q].x += wgt.x * s.x - wgt.y * s.y;
            acc[q].y += wgt.x * s.y + wgt.y * s.x;
        }
        __syncthreads();
    }
    for (int q = threadIdx.x; q < NN + 2; q += blockDim.x) out[q] = acc[q];
}

// ---------------------------------------------------------------------------
// The same for N <= 8 and at most two slots per state, with the lanes of
// heom_dmma_stage: lane 4r + t reads its two sectors of the neighbours along
// the baths of state r.  Of the bath terms it keeps theta-independent sums per
// slot -- <a, row and column terms> scaled by sqrt(n) or sqrt(n+1) -- and the
// derivatives of the coefficients enter once per launch and factor.  The next
// ADO's indices are read one ADO ahead: one round trip per ADO is exposed.
// Latency bounds it.  7 states, one slot, 6435 ADOs: 8.7 us a factor in launches
// of twelve, against 17 in launches of one with a lane per sector.
// ---------------------------------------------------------------------------
template <int N, int SLT>
__global__ void __launch_bounds__(kCtaWarps * 32, 2) heom_row_grad(const __grid_constant__ GradParams g)
{
    static_assert(N <= 8 && SLT <= 2, "row gradient handles N <= 8 and two slots");
    constexpr int P = pairs_of(N), NN = N * N, LD = N + 1;
    constexpr bool ODD = (N & 1) != 0;
    extern __shared__ __align__(128) unsigned char smem[];
    const int W = g.W;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double2* At = reinterpret_cast<double2*>(smem + warp * grad_warp_bytes(N)); // [N][N+1]
    double2* Wt = At + N * LD;
    double2* acc = reinterpret_cast<double2*>(smem + kCtaWarps * grad_warp_bytes(N)); // [NN+2]

    // ---- this lane's place (heom_dmma_stage) ----
    const int r = lane >> 2, t = lane & 3;
    const int odd = row_owned(r, t);
    const bool dga = t == (r >> 1) && !(r & 1), dgb = t == (r >> 1) && (r & 1);
    const int ps0 = opaque(g.rt.pos[lane][0]), ps1 = opaque(g.rt.pos[lane][1]);
    const int pso = odd ? ps1 : ps0, psg = odd ? ps0 : ps1;
    const bool owner = pso >= 0, holds = psg >= 0;
    const int co = 2 * t + odd, cg = 2 * t + 1 - odd;
    const int i2 = dga ? (r + 1 < N ? r + 1 : r) : co, j2 = dga ? i2 : r; // second element of the owned sector
    const bool twin = ODD && dga && r == N - 1;                            // padding half
    const int no_o = owner ? 0 : -1, no_g = holds ? 0 : -1;
    const int no_co = dga ? -1 : no_o, no_cg = dgb ? -1 : no_g;
    // tile positions: owned sector's halves, row and column element of the handed-over one
    const int q1 = owner ? r * LD + co : 0, q2 = owner ? i2 * LD + j2 : 0;
    const int gr = holds ? r * LD + cg : 0, gc = holds ? (dgb ? gr : cg * LD + r) : 0;
    int sl[SLT];
#pragma unroll
    for (int q = 0; q < SLT; ++q) sl[q] = (r < N && q < g.SL) ? g.slots[r * g.SL + q] : -1;
    auto el = [&](const double2* T, int i, int j) {
        return (N == 8 || (i < N && j < N)) ? T[i * LD + j] : make_double2(0.0, 0.0);
    };
    auto conj_mac = [](double2& s, const double2 a, const double2 w) { // s += conj(a) w
        s.x = fma(a.x, w.x, s.x);
        s.x = fma(a.y, w.y, s.x);
        s.y = fma(a.x, w.y, s.y);
        s.y = fma(-a.y, w.x, s.y);
    };

    const int inst = blockIdx.x / g.blocks_per_inst, jb = blockIdx.x - inst * g.blocks_per_inst;
    const unsigned stride = (unsigned)g.blocks_per_inst * kCtaWarps, end = (unsigned)g.inst_base[inst + 1];
    const unsigned begin = (unsigned)g.inst_base[inst] + (unsigned)jb * kCtaWarps + warp;
    const int recb = rec_bytes(g.NW, g.TWB);
    double2* const out = g.partial + (int64_t)blockIdx.x * (NN + 2);
    for (int q = threadIdx.x; q < NN + 2; q += blockDim.x) acc[q] = out[q];

    for (int f = 0; f < g.factors; ++f) {
        const double2* a_in = g.a + f * g.a_step;
        const double2* w_in = g.w + f * g.w_step;
        const double2 z0 = make_double2(0.0, 0.0);
        double zr0 = 0.0, zr1 = 0.0, zi0 = 0.0, zi1 = 0.0; // Z(r, 2t), Z(r, 2t+1)
        double2 sp[SLT], si[SLT], sj[SLT], y1 = z0, y2 = z0, sd = z0;
#pragma unroll
        for (int q = 0; q < SLT; ++q) sp[q] = si[q] = sj[q] = z0;
        int2 pm[SLT];
        int nn[SLT];
        auto index = [&](unsigned u) {
            const unsigned char* rec = g.rec + (int64_t)u * recb;
#pragma unroll
            for (int q = 0; q < SLT; ++q) {
                pm[q] = make_int2(-1, -1);
                nn[q] = 0;
                if (g.want_bath && sl[q] >= 0 && u < end) {
                    pm[q] = __ldg(reinterpret_cast<const int2*>(rec) + sl[q]);
                    nn[q] = rec[g.NW * 4 + sl[q]];
                }
            }
        };
        index(begin);
        for (unsigned u = begin; u < end; u += stride) {
            double2 a1 = z0, a2 = z0, w1 = z0, w2 = z0;
            double2 xo[2], xg[2]; // minus neighbour
            const int64_t o = (int64_t)u * (2 * P);
            if (owner) {
                ld256(a_in + o + 2 * pso, a1, a2);
                ld256(w_in + o + 2 * pso, w1, w2);
            }
            const double dps = g.dpss[u];
            int2 cm[SLT];
            int cn[SLT];
#pragma unroll
            for (int q = 0; q < SLT; ++q) {
                cm[q] = pm[q];
                cn[q] = nn[q];
            }
            auto minus = [&](int q) {
                const int64_t om = (int64_t)cm[q].y * (2 * P);
                ld256_if(cm[q].y | no_o, w_in + om + 2 * (owner ? pso : 0), xo[0], xo[1]);
                ld256_if(cm[q].y | no_g, w_in + om + 2 * (holds ? psg : 0), xg[0], xg[1]);
            };
            minus(0);
            index(u + stride);
            if (owner) {
                At[q1] = a1;
                At[q2] = a2;
                Wt[q1] = w1;
                Wt[q2] = w2;
            }
            __syncwarp();
            // Z(k,l) = sum_i w(i,k) conj(a(i,l)) - sum_j conj(a(k,j)) w(l,j):
            //   Re Z = Wr^T Ar + Wi^T Ai - Ar Wr^T - Ai Wi^T, Im Z = Wi^T Ar - Wr^T Ai - Ar Wi^T + Ai Wr^T
            if (g.want_h) {
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                    if (4 * s >= N) continue;
                    const int k0 = 4 * s + t;
                    const double2 wT = el(Wt, k0, r); // A operand of W^T A: W(4s+t, r)
                    const double2 aB = el(At, k0, r); // B operand of W^T A: A(4s+t, r)
                    const double2 aA = el(At, r, k0); // A operand of A W^T: A(r, 4s+t)
                    const double2 wB = el(Wt, r, k0); // B operand of A W^T: W(r, 4s+t)
                    dmma(zr0, zr1, wT.x, aB.x);
                    dmma(zr0, zr1, wT.y, aB.y);
                    dmma(zr0, zr1, -aA.x, wB.x);
                    dmma(zr0, zr1, -aA.y, wB.y);
                    dmma(zi0, zi1, wT.y, aB.x);
                    dmma(zi0, zi1, -wT.x, aB.y);
                    dmma(zi0, zi1, -aA.x, wB.y);
                    dmma(zi0, zi1, aA.y, wB.x);
                }
            }
            if (g.want_bath) {
                // same term of the owned elements (a padding half counts once)
                double2 v1 = z0, v2 = z0;
                conj_mac(v1, a1, w1);
                if (!twin) conj_mac(v2, a2, w2);
                y1.x += v1.x;
                y1.y += v1.y;
                y2.x += v2.x;
                y2.y += v2.y;
                sd.x = fma(dps, v1.x + v2.x, sd.x);
                sd.y = fma(dps, v1.y + v2.y, sd.y);
                const double2 ar = At[gr], ac = At[gc]; // handed-over sector: row and column element
#pragma unroll
                for (int q = 0; q < SLT; ++q) {
                    if (q > 0) minus(q);
                    if (cm[q].y >= 0) {
                        const double s = g.sq[cn[q]];
                        double2 vi = z0, vj = z0;
                        if (owner) {
                            conj_mac(vi, a1, xo[0]);
                            conj_mac(vj, dga ? a1 : a2, dga ? xo[0] : xo[1]);
                        }
                        if (holds) {
                            conj_mac(vi, ar, xg[1]);
                            conj_mac(vj, ac, dgb ? xg[1] : xg[0]);
                        }
                        si[q].x = fma(s, vi.x, si[q].x);
                        si[q].y = fma(s, vi.y, si[q].y);
                        sj[q].x = fma(s, vj.x, sj[q].x);
                        sj[q].y = fma(s, vj.y, sj[q].y);
                    }
                    if (cm[q].x >= 0) {
                        const int64_t op = (int64_t)cm[q].x * (2 * P);
                        ld256_if(no_co, w_in + op + 2 * (owner ? pso : 0), xo[0], xo[1]);
                        ld256_if(no_cg, w_in + op + 2 * (holds ? psg : 0), xg[0], xg[1]);
                        const double s = g.sq[cn[q] + 1];
                        double2 vr = z0, vc = z0; // row elements with +i, column elements with -i
                        if (no_co >= 0) {
                            conj_mac(vr, a1, xo[0]);
                            conj_mac(vc, a2, xo[1]);
                        }
                        if (no_cg >= 0) {
                            conj_mac(vr, ar, xg[1]);
                            conj_mac(vc, ac, xg[0]);
                        }
                        sp[q].x = fma(s, vc.y - vr.y, sp[q].x); // i (vr - vc)
                        sp[q].y = fma(s, vr.x - vc.x, sp[q].y);
                    }
                }
            }
            __syncwarp();
        }
        // the coefficients' derivatives, then the block's sum in a fixed order, times the factor's weight
        double2* mine = At; // [NN+2], where the warp's tiles were
        if (r < N && 2 * t < N) mine[r * N + 2 * t] = make_double2(zr0, zi0);
        if (r < N && 2 * t + 1 < N) mine[r * N + 2 * t + 1] = make_double2(zr1, zi1);
        double2 d[2] = {z0, sd}; // lambda, gamma
#pragma unroll
        for (int th = 0; th < 2; ++th) {
            if (g.want_bath && owner) {
                cmac(d[th], g.dg0[th * NN + r * N + co], y1);
                cmac(d[th], g.dg0[th * NN + i2 * N + j2], y2);
            }
#pragma unroll
            for (int q = 0; q < SLT; ++q) {
                if (!g.want_bath || sl[q] < 0) continue;
                const double2* kh = g.dkhat + th * 3 * W + sl[q];
                const double c = g.dchat[th * W + sl[q]];
                d[th].x = fma(c, sp[q].x, d[th].x);
                d[th].y = fma(c, sp[q].y, d[th].y);
                cmac(d[th], kh[0], si[q]);
                cmac(d[th], kh[W], sj[q]);
            }
            for (int off = 16; off > 0; off >>= 1) {
                d[th].x += __shfl_down_sync(0xffffffffu, d[th].x, off);
                d[th].y += __shfl_down_sync(0xffffffffu, d[th].y, off);
            }
            if (lane == 0) mine[NN + th] = d[th];
        }
        __syncthreads();
        const double2 wgt = g.weight[(g.factor0 - f) & 3];
        for (int q = threadIdx.x; q < NN + 2; q += blockDim.x) {
            double2 s = z0;
            for (int v = 0; v < kCtaWarps; ++v) {
                const double2 m = reinterpret_cast<const double2*>(smem + v * grad_warp_bytes(N))[q];
                s.x += m.x;
                s.y += m.y;
            }
            acc[q].x += wgt.x * s.x - wgt.y * s.y;
            acc[q].y += wgt.x * s.y + wgt.y * s.x;
        }
        __syncthreads();
    }
    for (int q = threadIdx.x; q < NN + 2; q += blockDim.x) out[q] = acc[q];
}


// y[top of instance k] += w * O_k (O_k row-major n x n complex, obs =
// [instances][n*n]), pair layout; block k.  w = weights[*base + j] (a device
// offset, so one captured graph serves every segment).
__global__ void heom_add_top(double2* __restrict__ y, const double2* __restrict__ obs_all,
                             const int16_t* __restrict__ pe, const int64_t* __restrict__ tops, int n, int P,
                             const double* __restrict__ weights, const int64_t* __restrict__ base, int64_t j)
{
    const double weight = weights[*base + j];
    if (weight == 0.0) return;
    const int64_t top = tops[blockIdx.x];
    const double2* obs = obs_all + (int64_t)blockIdx.x * n * n;
    for (int pr = threadIdx.x; pr < P; pr += blockDim.x) {
        const int e1 = pe[2 * pr], e2 = pe[2 * pr + 1];
        double2& h1 = y[(top * P + pr) * 2];
        double2& h2 = y[(top * P + pr) * 2 + 1];
        h1.x += weight * obs[e1].x;
        h1.y += weight * obs[e1].y;
        if (e2 != e1) {
            h2.x += weight * obs[e2].x;
            h2.y += weight * obs[e2].y;
        } else {
            h2 = h1; // padding half mirrors its element
        }
    }
}

// ---------------------------------------------------------------------------
// Time-dependent Hamiltonian (the e_field pre-evaluate action of the
// reference, e_field.hpp:63-85): H(t) = H - E(t) D- - conj(E(t)) D+ with
// E(t) = sum over the pulses of e0 exp(-(t - tc)^2 / (2 w^2)) exp(i (phi + omega t)).
// One block builds the operand tables of H(t) for `nt` times t0 + c_s dt of
// every instance: stage times c = (0, 1/2, 1) of an RK4 step when `time` is
// given (t0 = *time, then *time += dt), or the single time t0 of an explicit
// evaluation.
// ---------------------------------------------------------------------------
struct Pulse {
    double e0, tc, w, omega, phi;
};
struct FieldParams {
    const double2* h0;     // [K][N*N] H / hbar of every instance
    const double2* dplus;  // [N*N] D+ / hbar
    const double2* dminus; // [N*N] D- / hbar
    Pulse pulse[2];        // pump, probe
    double* time;          // step mode: device time of the propagation state (advanced by dt)
    double t0, dt;         // explicit mode: the evaluation time t0 (time == nullptr)
    double2* hs_t;         // [nt][K][N*N]
    double* frag_t;        // [nt][K][frag_doubles(N)]
    int K, N, nt;
};

__device__ inline double2 field_at(const FieldParams& f, double t)
{
    double er = 0.0, ei = 0.0;
    for (int q = 0; q < 2; ++q) {
        const Pulse& pl = f.pulse[q];
        const double d = t - pl.tc;
        const double env = pl.e0 * exp(-d * d / (2.0 * pl.w * pl.w));
        double sn, cs;
        sincos(pl.phi + pl.omega * t, &sn, &cs);
        er += env * cs;
        ei += env * sn;
    }
    return make_double2(er, ei);
}

__global__ void heom_field_tables(const FieldParams f)
{
    const int N = f.N, NN = N * N;
    const double t0 = f.time ? *f.time : f.t0;
    const double cst[3] = {0.0, 0.5, 1.0};
    for (int s = 0; s < f.nt; ++s) {
        const double2 E = field_at(f, t0 + cst[s] * f.dt);
        for (int k = 0; k < f.K; ++k) {
            double2* hs = f.hs_t + ((size_t)s * f.K + k) * NN;
            for (int q = threadIdx.x; q < NN; q += blockDim.x) {
                const double2 h = f.h0[(size_t)k * NN + q], dm = f.dminus[q], dp = f.dplus[q];
                // H - E D- - conj(E) D+
                const double re = h.x - (E.x * dm.x - E.y * dm.y) - (E.x * dp.x + E.y * dp.y);
                const double im = h.y - (E.x * dm.y + E.y * dm.x) - (E.x * dp.y - E.y * dp.x);
                hs[q] = make_double2(re, im);
            }
            __syncthreads();
            {
                const int fd = frag_doubles(N), nb = frag_blocks(N), ns = frag_slices(N);
                for (int q = threadIdx.x; q < fd; q += blockDim.x) {
                    // operand fragments as in the host tables ([kind][block][k-slice][lane], frag_index)
                    const int l = q & 31, part = q >> 5, sl = part % ns, b = (part / ns) % nb, kind = part / (ns * nb);
                    const int r = 8 * b + (l >> 2), c = frag_col(N, sl, l & 3);
                    double v = 0.0;
                    if (r < N && c < N) {
                        const double2 hcr = hs[c * N + r], hrc = hs[r * N + c];
                        v = kind == 0 ? hcr.x : kind == 1 ? hcr.y : kind == 2 ? -hrc.x : -hrc.y;
                    }
                    f.frag_t[((size_t)s * f.K + k) * fd + q] = v;
                }
            }
            __syncthreads();
        }
    }
    if (f.time && threadIdx.x == 0) *f.time = t0 + f.dt;
}

// ---------------------------------------------------------------------------
// Hierarchy arithmetic (hierarchy_arithmetic_{add,subtract,scale,dot_product,
// mmult_left,mmult_right}.cl) on whole state buffers in the pair layout, in
// the reference's operation order (complex products as a.x*b.x - a.y*b.y,
// sums in k order, no contraction).  out may alias a or b.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double2 cmul_rn(double2 a, double2 b)
{
    return make_double2(__dsub_rn(__dmul_rn(a.x, b.x), __dmul_rn(a.y, b.y)),
                        __dadd_rn(__dmul_rn(a.x, b.y), __dmul_rn(a.y, b.x)));
}

// op 0: a + b, 1: a - b, 2: a * conj(b), 3: f * a
__global__ void heom_hier_elementwise(double2* out, const double2* a, const double2* b, double2 f, int64_t len, int op)
{
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < len; e += stride) {
        const double2 x = a[e];
        double2 r;
        if (op == 0) {
            const double2 y = b[e];
            r = make_double2(__dadd_rn(x.x, y.x), __dadd_rn(x.y, y.y));
        } else if (op == 1) {
            const double2 y = b[e];
            r = make_double2(__dsub_rn(x.x, y.x), __dsub_rn(x.y, y.y));
        } else if (op == 2) {
            const double2 y = b[e];
            r = cmul_rn(x, make_double2(y.x, -y.y));
        } else {
            r = cmul_rn(f, x);
        }
        out[e] = r;
    }
}

// every ADO: out_u = M a_u (left) or a_u M (right); one warp per ADO, the
// tile staged in shared memory ([warp][N*N] double2)
__global__ void heom_hier_mmult(double2* out, const double2* a, const double2* __restrict__ m,
                                const int16_t* __restrict__ pe, int64_t nodes, int n, int P, int left)
{
    extern __shared__ __align__(128) unsigned char smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, NN = n * n;
    double2* t = reinterpret_cast<double2*>(smem) + warp * 2 * NN;
    double2* r = t + NN;
    const int64_t stride = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t u = (int64_t)blockIdx.x * (blockDim.x >> 5) + warp; u < nodes; u += stride) {
        for (int pr = lane; pr < P; pr += 32) {
            t[pe[2 * pr]] = a[(u * P + pr) * 2];
            t[pe[2 * pr + 1]] = a[(u * P + pr) * 2 + 1];
        }
        __syncwarp();
        for (int q = lane; q < NN; q += 32) {
            const int i = q / n, j = q - i * n;
            double2 v = make_double2(0.0, 0.0);
            for (int k = 0; k < n; ++k) {
                const double2 p = left ? cmul_rn(m[i * n + k], t[k * n + j]) : cmul_rn(t[i * n + k], m[k * n + j]);
                v = make_double2(__dadd_rn(v.x, p.x), __dadd_rn(v.y, p.y));
            }
            r[q] = v;
        }
        __syncwarp();
        for (int pr = lane; pr < P; pr += 32) {
            out[(u * P + pr) * 2] = r[pe[2 * pr]];
            out[(u * P + pr) * 2 + 1] = r[pe[2 * pr + 1]];
        }
        __syncwarp();
    }
}

// Frobenius norm squared of every ADO, sum |sigma(i,j)|^2 (hierarchy_norm.cl:15-45),
// written at the ADO's reference index.  One warp per ADO; a padding half of
// an odd diagonal pair counts once.
__global__ void heom_hierarchy_norm(double* __restrict__ norms, const double2* __restrict__ y,
                                    const int64_t* __restrict__ ref_of_int, const int16_t* __restrict__ pe,
                                    int64_t nodes, int P)
{
    const int lane = threadIdx.x & 31;
    const int64_t stride = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t u = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); u < nodes; u += stride) {
        double acc = 0.0;
        for (int pr = lane; pr < P; pr += 32) {
            const double2 a = y[(u * P + pr) * 2], b = y[(u * P + pr) * 2 + 1];
            acc += a.x * a.x + a.y * a.y;
            if (pe[2 * pr + 1] != pe[2 * pr]) acc += b.x * b.x + b.y * b.y;
        }
        for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
        if (lane == 0) norms[ref_of_int[u]] = acc;
    }
}

// Sets *flag (mapped host memory) when any element is not finite.
__global__ void heom_check_finite(const double* __restrict__ y, int64_t len, int* flag)
{
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    int bad = 0;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < len; e += stride)
        bad |= !isfinite(y[e]);
    if (__syncthreads_or(bad) && threadIdx.x == 0) *static_cast<volatile int*>(flag) = 1;
}

} // namespace heomk

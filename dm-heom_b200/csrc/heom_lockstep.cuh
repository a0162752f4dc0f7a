// heom_lockstep.cuh -- sm_100a stage kernel of a lockstep ensemble class.
//
// A lockstep class holds K >= 8 instances of one hierarchy shape (same states,
// baths, Matsubara terms and depth: the realisations of a static-disorder
// ensemble) with the state stored instance-minor: sector p of ADO u of
// instance k at ((u * P + p) * Kp + k) * 32 bytes, Kp = K rounded up to 32.
// Each stage evaluates the same per-element derivative as heom_dmma_stage
// (heom_ode.cl:24-451, the RK4 write fused), in the same operation order, so
// that every instance's results are those of a single-instance solve; what
// changes is the traffic: a sector row of 32 instances is one coalesced
// 1-KB read, and the neighbour indices, coefficients and site bookkeeping of
// an ADO are resolved once for all of its instances.

#pragma once

#include "heom_kernels.cuh"

namespace heomk {

struct LockParams {
    PairParams p;     // in/out/y/acc in the lockstep layout; records of one instance; hfrag [K][256]
    LaneTab lt;
    CoefTabs ct;
    int K;            // instances
    int Kp;           // instance stride (K rounded up to 32)
    int64_t nodes;    // ADOs of every instance
};

constexpr int kLockWarps = 8;
// one slot of one site at the current ADO: its neighbour rows and coefficients
struct __align__(16) LockSlot {
    int64_t op, om;   // byte offsets of the rows of ADO n + e (plus) and n - e (minus); -1: absent
    double2 kap[3];   // minus-side coefficients: the three kappa-hat values of the slot times sqrt(n)
    double c;         // plus-side coefficient chat * sqrt(n + 1)
    double pad;
};
// one pair sector, in the order in which the warps take them: its sites and same-term values
struct __align__(16) LockSector {
    int sa, sb, diag, ps;  // sites of side 0 and side 1 (element i1, then j1 or, diagonal, i2); the sector
    double2 g1, g2;        // gamma0 of its two elements
    int twin, pad[3];      // 1: the second half is the padding half, the first's copy
};
__host__ __device__ inline int lock_row_bytes(int NW, int TWB) { return rec_bytes(NW, TWB); }
// rows of the commutator tile: the sectors, and for N < 8 one for elements outside the N x N block
__host__ __device__ constexpr int lock_comm_rows(int P) { return P < 32 ? P + 1 : 32; }
__host__ inline size_t lockstep_smem_bytes(int P, int W, int NW, int TWB, int LS)
{
    return (size_t)dmma_lut_bytes(W, LS) + 2 * (size_t)P * 32 * 32 /* two tiles */ +
           (size_t)lock_comm_rows(P) * 32 * 32 /* commutators */ + 32 * sizeof(LockSector) + 32 * sizeof(LockSlot) +
           2 * (size_t)lock_row_bytes(NW, TWB);
}

// 32 bytes at base + off (bytes) when off >= 0; otherwise a and b keep what they hold: the test, the
// address and the load in one asm block
__device__ __forceinline__ void ld256_at(const double2* base, int64_t off, double2& a, double2& b)
{
    asm("{\n .reg .pred q;\n .reg .b64 ad;\n setp.ge.s64 q, %5, 0;\n add.s64 ad, %4, %5;\n"
        " @q ld.global.v4.f64 {%0,%1,%2,%3}, [ad];\n}\n"
        : "+d"(a.x), "+d"(a.y), "+d"(b.x), "+d"(b.y)
        : "l"(base), "l"(off));
}
// 32 bytes through the coherent path, schedulable: the stage kernel stores to the same address only
// values computed from the loaded ones, which orders the load first
__device__ __forceinline__ void ld256_co(const double2* src, double2& a, double2& b)
{
    asm("ld.global.v4.f64 {%0,%1,%2,%3}, [%4];\n" : "=d"(a.x), "=d"(a.y), "=d"(b.x), "=d"(b.y) : "l"(src));
}

// Two CTAs of 8 warps per SM. CTA b keeps the instance block b % (Kp / 32)
// and sweeps the ADOs u = b / (Kp / 32), + gridDim / (Kp / 32), ...; the next
// ADO's tiles and rows are copied (cp.async) while the current one runs.
// Phase A: warp w forms the commutator of instances w, w + 8, w + 16, w + 24
// of the block (real symmetric H: their fragments stay in registers, the A
// operand being -hb exactly); the last warp first resolves every slot of every
// site at this ADO into a table (neighbour rows, coefficients), so that phase
// B's sectors read broadcast entries. Phase B: one warp per sector, a lane per
// instance; every global read of a sector (the neighbour rows of both sides,
// y and acc) is issued, predicated, before its arithmetic.
template <int N, int HK, int SLT>
__global__ void __launch_bounds__(kLockWarps * 32, 2) heom_lockstep_stage(const __grid_constant__ LockParams lp)
{
    static_assert(N <= 8 && N * SLT <= 32, "lockstep stage handles N <= 8");
    constexpr int P = pairs_of(N);
    constexpr int IPW = 32 / kLockWarps;  // instances per warp in phase A
    constexpr int SB = SLT <= 1 ? 2 : 1; // sides whose neighbour rows are read in one batch
    constexpr int QB = SLT < 2 ? SLT : 2; // slots read in one batch
    constexpr int TW = kLockWarps - 1;   // the warp that builds the site table
    const PairParams& p = lp.p;
    extern __shared__ __align__(128) unsigned char smem[];
    const int W = p.W, LS = p.LS, SL = p.SL;
    grid_launch_dependents();
    double2* s_kh = reinterpret_cast<double2*>(smem);
    double2* s_sq = s_kh + 3 * W;
    double* s_ch = reinterpret_cast<double*>(s_sq + LS + 1);
    for (int q = threadIdx.x; q < 3 * W; q += blockDim.x) s_kh[q] = lp.ct.khat[q];
    for (int q = threadIdx.x; q < W; q += blockDim.x) s_ch[q] = lp.ct.chat[q];
    for (int q = threadIdx.x; q <= LS; q += blockDim.x)
        s_sq[q] = make_double2(lp.ct.sq[q], q < LS ? lp.ct.sq[q + 1] : 0.0);
    unsigned char* base = smem + dmma_lut_bytes(W, LS);
    double2* tiles = reinterpret_cast<double2*>(base);      // [2][P][32] sectors (2 double2 each)
    double2* ctile = tiles + 2 * 2 * P * 32;                 // [P][32] commutator values, one row more for N < 8
    LockSector* sectors = reinterpret_cast<LockSector*>(ctile + 2 * lock_comm_rows(P) * 32);
    LockSlot* slots = reinterpret_cast<LockSlot*>(sectors + 32);
    unsigned char* rows0 = reinterpret_cast<unsigned char*>(slots + 32);
    const int rowb = lock_row_bytes(p.NW, p.TWB);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kblocks = lp.Kp >> 5;
    const int kb = blockIdx.x % kblocks;
    const int64_t ustep = gridDim.x / kblocks;
    const int64_t Kp = lp.Kp;
    const int64_t PK2 = (int64_t)P * Kp * 2; // double2 elements of one ADO (all instances)

    if (threadIdx.x < P) {
        const int ps = lp.lt.ord[threadIdx.x], e1 = lp.lt.e1[ps], e2 = lp.lt.e2[ps];
        const int i1 = e1 / N, j1 = e1 - i1 * N, i2 = e2 / N;
        LockSector sc;
        sc.sa = i1;
        sc.diag = i1 == j1;
        sc.sb = sc.diag ? i2 : j1;
        sc.ps = ps;
        sc.g1 = p.gamma0[e1];
        sc.g2 = p.gamma0[e2];
        sc.twin = e1 == e2 ? 1 : 0;
        sc.pad[0] = sc.pad[1] = sc.pad[2] = 0;
        sectors[threadIdx.x] = sc;
    }

    // real symmetric H: hb of this warp's instances for the whole sweep
    double hbk[IPW][2];
#pragma unroll
    for (int j = 0; j < IPW; ++j) {
        const int k = kb * 32 + warp + kLockWarps * j;
#pragma unroll
        for (int s = 0; s < 2; ++s)
            hbk[j][s] = (HK != H_GENERIC && k < lp.K) ? __ldg(p.hfrag + (size_t)k * 256 + 32 * s + lane) : 0.0;
    }

    const int fs0 = opaque(lp.lt.fs[lane][0]), fs1 = opaque(lp.lt.fs[lane][1]);
    const int ha0 = opaque(lp.lt.ha[lane][0]), ha1 = opaque(lp.lt.ha[lane][1]);
    const int r = lane >> 2, t = lane & 3;
    // Phase A offsets (double2, from a tile buffer) of this lane's operands for the warp's first
    // instance; its instance warp + 8 j adds 16 j, since the column swizzle k ^ (p & 3) changes
    // bits 0-1 of k only. A lane outside the N x N block reads what a lane of its quarter warp inside it
    // reads (LaneTab), which costs no wavefront: its partner fragment of H is zero, so it adds only zeros
    // as long as the value is finite, and it is one of the same instance, so that a realisation that has
    // diverged stays by itself.
    // Shared tiles store half h of instance column k at position h ^ ((k >> 2) & 1): a warp's
    // 16-byte accesses to one half of 32 columns then cover all eight 16-byte bank groups.
    const int hw = (warp >> 2) & 1; // (k >> 2) & 1 of the warp's phase A instances
    int oa[2], ob[2];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        const int fs = s == 0 ? fs0 : fs1, ha = s == 0 ? ha0 : ha1;
        const int row = (fs * 32 + (warp ^ (fs & 3))) * 2;
        oa[s] = row + (ha ^ hw);
        ob[s] = row + (r < N && r == 2 * t + s ? ha ^ hw : ha ^ 1 ^ hw); // diagonal: its own transpose
    }
    // the MMA result is the lane's own row elements (r, 2t), (r, 2t+1): the commutator of element (r, 2t+s) goes
    // where the A operand of slice s was read (elements outside the N x N block: a row that is not read)
    const int oc0 = r < N && 2 * t < N ? oa[0] : P * 64, oc1 = r < N && 2 * t + 1 < N ? oa[1] : P * 64;
    const int hk = (lane >> 2) & 1; // phase B: position of half 0 of this lane's instance
    // the slot of site (lane / SLT) that lane of the table warp resolves
    const int tsite = lane / SLT, tq = lane - tsite * SLT;
    const int tsl = (warp == TW && tsite < N && tq < SL) ? __ldg(p.slots + tsite * SL + tq) : -1;
    const int tpos = tsl >= 0 ? lp.ct.pos[tsl] : 0;
    // this thread's 16-byte pieces of a tile copy: sectors pp0, pp0 + 4, ... of instance column pk
    const int pp0 = threadIdx.x >> 6, pk = (threadIdx.x >> 1) & 31, ph = threadIdx.x & 1;
    const int dst0 = (pp0 * 32 + (pk ^ (pp0 & 3))) * 2 + (ph ^ ((pk >> 2) & 1));
    const int64_t src0 = ((int64_t)pp0 * Kp + pk) * 2 + ph + (int64_t)kb * 64;

    // asynchronous copies of ADO u's tiles (this block's 32 instances) and rows into buffer b
    auto prefetch = [&](int64_t u, int b) {
        double2* dst = tiles + b * 2 * P * 32 + dst0;
        const double2* src = p.in + u * PK2 + src0;
        for (int pp = pp0; pp < P; pp += 4, dst += 4 * 64, src += 8 * Kp) cp_async16(dst, src);
        unsigned char* rows = rows0 + b * rowb;
        const int recb = rec_bytes(p.NW, p.TWB);
        for (int q = threadIdx.x * 16; q < recb; q += blockDim.x * 16) cp_async16(rows + q, p.rec + u * recb + q);
    };

    const int kl = kb * 32 + lane;
    const bool live = kl < lp.K;
    const bool read_acc = p.use_acc && !p.acc_init;
    grid_wait(); // the state is written by the kernels before this one
    int64_t u = blockIdx.x / kblocks;
    int cur = 0;
    if (u < lp.nodes) prefetch(u, 0);
    for (; u < lp.nodes; u += ustep, cur ^= 1) {
        cp_async_wait_all();
        __syncthreads();
        // the next ADO's copies fly while this one runs (its buffer was last read before the barrier)
        if (u + ustep < lp.nodes) prefetch(u + ustep, cur ^ 1);
        const double2* tile = tiles + cur * 2 * P * 32;
        const unsigned char* rows = rows0 + cur * rowb;
        const unsigned char* tu = rows + ((p.NW * 4 + 15) & ~15);
        const double2 pss = *reinterpret_cast<const double2*>(tu + ((p.TWB + 15) & ~15));

        // ---- the site table of this ADO ----
        if (warp == TW && lane < N * SLT) {
            LockSlot e;
            e.pad = 0.0;
            if (tsl >= 0) {
                const int2 pm = reinterpret_cast<const int2*>(rows)[tsl];
                const double2 sqp = s_sq[tu[tsl]];
                e.op = pm.x >= 0 ? pm.x * PK2 * 16 : -1;
                e.om = pm.y >= 0 ? pm.y * PK2 * 16 : -1;
                e.c = s_ch[tpos] * sqp.y;
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    const double2 v = s_kh[q * W + tpos];
                    e.kap[q] = make_double2(v.x * sqp.x, v.y * sqp.x);
                }
            } else {
                e.op = e.om = -1;
                e.c = 0.0;
                e.kap[0] = e.kap[1] = e.kap[2] = make_double2(0.0, 0.0);
            }
            slots[lane] = e;
        }

        // ---- A: commutator of every instance of the block ----
        {
            double gf[HK == H_GENERIC ? IPW : 1][2][4];
            if (HK == H_GENERIC) {
#pragma unroll
                for (int j = 0; j < IPW; ++j) {
                    const int kj = kb * 32 + warp + kLockWarps * j;
                    const double* f = p.hfrag + (size_t)(kj < lp.K ? kj : 0) * 256 + lane;
#pragma unroll
                    for (int s = 0; s < 2; ++s)
#pragma unroll
                        for (int c = 0; c < 4; ++c) gf[HK == H_GENERIC ? j : 0][s][c] = __ldg(f + 32 * (2 * c + s));
                }
            }
#pragma unroll
            for (int j0 = 0; j0 < IPW; j0 += 2) {
                double cr[2][2], ci[2][2]; // the two instances' accumulators
#pragma unroll
                for (int jj = 0; jj < 2; ++jj) {
                    const int j = j0 + jj;
                    double hb_r[2], hb_i[2], ha_r[2], ha_i[2];
#pragma unroll
                    for (int s = 0; s < 2; ++s) {
                        if (HK == H_GENERIC) {
                            hb_r[s] = gf[HK == H_GENERIC ? j : 0][s][0];
                            hb_i[s] = gf[HK == H_GENERIC ? j : 0][s][1];
                            ha_r[s] = gf[HK == H_GENERIC ? j : 0][s][2];
                            ha_i[s] = gf[HK == H_GENERIC ? j : 0][s][3];
                        } else {
                            hb_r[s] = hbk[j][s];
                            ha_r[s] = -hbk[j][s]; // -H(r, c) = -H(c, r): H is real symmetric
                            hb_i[s] = ha_i[s] = 0.0;
                        }
                    }
                    cr[jj][0] = cr[jj][1] = ci[jj][0] = ci[jj][1] = 0.0;
#pragma unroll
                    for (int s = 0; s < 2; ++s) {
                        const double2 A = tile[oa[s] + 16 * j], B = tile[ob[s] + 16 * j];
                        dmma(cr[jj][0], cr[jj][1], A.x, hb_r[s]);
                        dmma(ci[jj][0], ci[jj][1], A.y, hb_r[s]);
                        dmma(cr[jj][0], cr[jj][1], ha_r[s], B.x);
                        dmma(ci[jj][0], ci[jj][1], ha_r[s], B.y);
                        if (HK == H_GENERIC) {
                            dmma(cr[jj][0], cr[jj][1], -A.y, hb_i[s]);
                            dmma(ci[jj][0], ci[jj][1], A.x, hb_i[s]);
                            dmma(cr[jj][0], cr[jj][1], -ha_i[s], B.y);
                            dmma(ci[jj][0], ci[jj][1], ha_i[s], B.x);
                        }
                    }
                }
#pragma unroll
                for (int jj = 0; jj < 2; ++jj) {
                    const int j = j0 + jj;
                    ctile[oc0 + 16 * j] = make_double2(cr[jj][0], ci[jj][0]);
                    ctile[oc1 + 16 * j] = make_double2(cr[jj][1], ci[jj][1]);
                }
            }
        }
        __syncthreads();

        // ---- B: per sector, lane = instance ----
        for (int k = warp; k < P; k += kLockWarps) {
            const LockSector sc = sectors[k];
            const int ps = sc.ps;
            const bool diag = sc.diag != 0;
            const int64_t lofs = ((int64_t)ps * Kp + kl) * 2; // this lane's sector within an ADO
            const double2* in_l = p.in + lofs;
            const int64_t off = u * PK2 + lofs;
            double2 x1, x2, a1, a2, s1, s2;
            // terms of side 0 (the first half's row) and of side 1, for both halves of the sector; either half's
            // own row starts with its commutator and same term
            double2 A[2][2];
            A[0][1] = A[1][0] = make_double2(0.0, 0.0);
#pragma unroll
            for (int sd0 = 0; sd0 < 2; sd0 += SB) {
#pragma unroll
                for (int q0 = 0; q0 < SLT; q0 += QB) {
                    // neighbour rows of SB sides and QB slots (absent rows: no load, zeros)
                    double2 xp[SB][QB][2], xm[SB][QB][2];
#pragma unroll
                    for (int b = 0; b < SB; ++b) {
                        const LockSlot* es = slots + ((sd0 + b) == 0 ? sc.sa : sc.sb) * SLT + q0;
#pragma unroll
                        for (int q = 0; q < QB; ++q) {
                            const longlong2 o = *reinterpret_cast<const longlong2*>(&es[q].op);
                            ld256_at(in_l, o.y, xm[b][q][0], xm[b][q][1]);
                            ld256_at(in_l, diag ? -1 : o.x, xp[b][q][0], xp[b][q][1]);
                        }
                    }
                    if (sd0 == 0 && q0 == 0) {
                        if (p.y) ld256_co(p.y + off, x1, x2); // kernel parameters: uniform branches
                        if (read_acc) ld256_co(p.acc + off, a1, a2);
                        const int col = (ps * 32 + (lane ^ (ps & 3))) * 2;
                        s1 = tile[col + hk];
                        s2 = tile[col + (hk ^ 1)];
                        const double2 c1 = ctile[col + hk], c2 = ctile[col + (hk ^ 1 ^ sc.twin)];
                        A[0][0] = make_double2(-c1.y, c1.x); // i * (w H - H w) / hbar
                        A[1][1] = make_double2(-c2.y, c2.x);
                        cmac(A[0][0], make_double2(pss.x + sc.g1.x, pss.y + sc.g1.y), s1);
                        cmac(A[1][1], make_double2(pss.x + sc.g2.x, pss.y + sc.g2.y), s2);
                    }
#pragma unroll
                    for (int b = 0; b < SB; ++b) {
                        const int sd = sd0 + b;
                        const LockSlot* es = slots + (sd == 0 ? sc.sa : sc.sb) * SLT + q0;
                        // minus neighbours of the batch, then its plus neighbours (heom_dmma_stage's order)
#pragma unroll
                        for (int q = 0; q < QB; ++q) {
                            if (es[q].om < 0) continue; // warp-uniform
                            const double2 kd = es[q].kap[diag ? 2 : 0], kj = es[q].kap[1];
                            if (sd == 0) {
                                cmac(A[0][0], kd, xm[b][q][0]);
                                if (!diag) cmac(A[0][1], kj, xm[b][q][1]);
                            } else {
                                if (!diag) cmac(A[1][0], kj, xm[b][q][0]);
                                cmac(A[1][1], kd, xm[b][q][1]);
                            }
                        }
                        if (diag) continue; // the plus terms of a diagonal element's row and column cancel
#pragma unroll
                        for (int q = 0; q < QB; ++q) {
                            if (es[q].op < 0) continue;
                            const double c = sd == 0 ? es[q].c : -es[q].c;
                            const double2 t1 = xp[b][q][0], t2 = xp[b][q][1];
                            A[sd][0].x = fma(-c, t1.y, A[sd][0].x);
                            A[sd][0].y = fma(c, t1.x, A[sd][0].y);
                            A[sd][1].x = fma(c, t2.y, A[sd][1].x);
                            A[sd][1].y = fma(-c, t2.x, A[sd][1].y);
                        }
                    }
                }
            }
            const double2 L1 = make_double2(A[0][0].x + A[1][0].x, A[0][0].y + A[1][0].y);
            const double2 L2 = make_double2(A[0][1].x + A[1][1].x, A[0][1].y + A[1][1].y);
            if (!p.y) {
                x1 = s1;
                x2 = s2;
            }
            double2 o1 = p.use_x ? x1 : make_double2(0.0, 0.0), o2 = p.use_x ? x2 : make_double2(0.0, 0.0);
            cmac(o1, p.beta, L1);
            cmac(o2, p.beta, L2);
            st256_cs_if(live, p.out + off, o1, o2);
            if (p.use_acc) {
                if (!read_acc) {
                    a1 = s1;
                    a2 = s2;
                }
                cmac(a1, p.acc_beta, L1);
                cmac(a2, p.acc_beta, L2);
                st256_if(live, p.acc + off, a1, a2);
            }
        }
    }
    cp_async_wait_all(); // no copy left in flight when the CTA retires
}

} // namespace heomk

// Host-only check of the stage kernel's shared-memory carve-up and pair
// table (compiled by tests/test_layout.py with nvcc; runs on the CPU).
// Prints one line per problem: "bad ..." for any violation, then "ok N".
#include <cstdio>
#include "heom_kernels.cuh"
#include "pair_tables.inc"
#include "row_tables.inc"

// Extra wavefronts of the operand reads of one tile by the lanes 4r + t of a warp: row element (r, 2t+s), then column
// element (2t+s, r), for s = 0, 1; sector p's half h lies in 16-byte bank group 2p + h (mod 8). A lane of a diagonal
// element reads in its second read the element itself (the lockstep kernel) or, when it owns the diagonal sector, the
// sector's second element (the N <= 8 stage kernel). Lanes outside the tile read zeros elsewhere.
static int extra_wavefronts(int n, const signed char* e1, const signed char* e2, bool owner_reads_second)
{
    int sec[64], half[64], extra = 0;
    for (int p = heomk::pairs_of(n) - 1; p >= 0; --p) {
        sec[e2[p]] = p; half[e2[p]] = 1;
        sec[e1[p]] = p; half[e1[p]] = 0;
    }
    for (int q = 0; q < 4; ++q)
        for (int s = 0; s < 2; ++s)
            for (int which = 0; which < 2; ++which) {
                unsigned addr[8];
                int count = 0, most = 1;
                for (int r = 2 * q; r <= 2 * q + 1; ++r)
                    for (int t = 0; t < 4; ++t) {
                        const int c = 2 * t + s;
                        if (r >= n || c >= n) continue;
                        const int e = which ? c * n + r : r * n + c;
                        const bool second = which && r == c && s == 0 && owner_reads_second;
                        addr[count++] = 2 * sec[e] + (second ? 1 : half[e]);
                    }
                for (int a = 0; a < count; ++a) {
                    int same = 1; // different addresses in a's group
                    for (int b = 0; b < a; ++b) {
                        bool seen = addr[b] == addr[a];
                        for (int k = 0; k < b; ++k) seen = seen || addr[k] == addr[b];
                        if (!seen && addr[b] % 8 == addr[a] % 8) ++same;
                    }
                    most = same > most ? same : most;
                }
                extra += most - 1;
            }
    return extra;
}

int main()
{
    long checked = 0, bad = 0;
    for (int n = 1; n <= 16; ++n) {
        // pair table: every element covered exactly once (diagonal padding duplicate allowed)
        int seen[256] = {0};
        const int P = heomk::pairs_of(n);
        for (int p = 0; p < P; ++p) {
            int e1, e2, i, j, d;
            heomk::pair_elements(n, p, &e1, &e2, &i, &j, &d);
            if (e1 < 0 || e1 >= n * n || e2 < 0 || e2 >= n * n) { printf("bad pair range n=%d p=%d\n", n, p); ++bad; }
            seen[e1]++;
            if (e2 != e1) seen[e2]++;
            if (!d && !(i < j && e1 == i * n + j && e2 == j * n + i)) { printf("bad offdiag n=%d p=%d\n", n, p); ++bad; }
        }
        for (int e = 0; e < n * n; ++e)
            if (seen[e] != 1) { printf("bad coverage n=%d e=%d count=%d\n", n, e, seen[e]); ++bad; }
        for (int W = 1; W <= 64; ++W)
            for (int depth = 1; depth <= 40; ++depth) {
                const int LS = depth + 1, NW = (2 * W + 3) & ~3, TWB = (W + 15) & ~15;
                const heomk::PairSmem L = heomk::pair_smem_layout(n, W, NW, TWB, LS);
                // khat 3W double2, (sqrt(n), sqrt(n+1)) for n = 0..LS, chat W doubles
                if (3 * W * 16 + (LS + 1) * 16 + W * 8 > L.lut) { printf("bad lut n=%d W=%d LS=%d\n", n, W, LS); ++bad; }
                if (L.lut % 128 || L.slot % 16 || L.team % 16 || L.tile_off % 16 || L.nbr_off % 16 ||
                    L.tup_off % 16 || L.pss_off % 16 || L.xch_off % 16 || L.hand_off % 16 || L.gam_off % 16) { printf("bad slot n=%d W=%d\n", n, W); ++bad; }
                if (L.nbr_off - L.tile_off < n * heomk::tile_stride(n) * 16 || L.tup_off - L.nbr_off < NW * 4 ||
                    L.pss_off - L.tup_off < TWB || L.slot - L.pss_off < 16 || L.xch_off < 2 * L.slot ||
                    // two exchange tiles, two copies of the terms handed over ([2][threads]), gamma0 ([2][threads])
                    L.hand_off - L.xch_off < 2 * heomk::kXchBytes ||
                    L.gam_off - L.hand_off < 2 * 2 * heomk::team_warps(n) * 32 * 16 ||
                    L.team - L.gam_off < 2 * heomk::team_warps(n) * 32 * 16)
                    { printf("bad sizes n=%d W=%d\n", n, W); ++bad; }
                if (NW % 4 || NW < 2 * W || TWB % 16 || TWB < W) { printf("bad pads W=%d\n", W); ++bad; }
                ++checked;
            }
        // gradient kernels: a warp's sums fit where its tiles were, and two blocks an SM (228 KB, 1 KB of them the
        // system's for each block) at the widest tables that a handle takes
        if ((n * n + 2) * 16 > heomk::grad_warp_bytes(n)) { printf("bad gradient sums n=%d\n", n); ++bad; }
        if (2 * (heomk::grad_smem_bytes(n, 255, 251) + 1024) > 228 * 1024) { printf("bad gradient blocks n=%d\n", n); ++bad; }
        // team kernel: the sectors in the order of their owners' threads, every one of them once; a sector is held by
        // two threads, one of which owns it
        if (n > 8) {
            const int T = (n + 1) / 2;
            int owners[136] = {0}, covered[256] = {0};
            for (int r = 0; r < n; ++r)
                for (int t = 0; t < T; ++t) {
                    const int c = 2 * t + heomk::row_owned(r, t);
                    if (c >= n) continue;
                    const int pos = heomk::team_pos(n, r, t);
                    if (pos < 0 || pos >= P || owners[pos]++) { printf("bad owner position n=%d (%d,%d)\n", n, r, t); ++bad; continue; }
                    const int i2 = c == r ? (r + 1 < n ? r + 1 : r) : c, j2 = c == r ? i2 : r;
                    covered[r * n + c]++;
                    if (i2 * n + j2 != r * n + c) covered[i2 * n + j2]++;
                }
            for (int p = 0; p < P; ++p)
                if (!owners[p]) { printf("bad: no owner n=%d p=%d\n", n, p); ++bad; }
            for (int e = 0; e < n * n; ++e)
                if (covered[e] != 1) { printf("bad owner coverage n=%d e=%d count=%d\n", n, e, covered[e]); ++bad; }
        }
        // tile positions: inside the row, one per element
        {
            int used[16 * 20] = {0};
            for (int i = 0; i < n; ++i)
                for (int k = 0; k < n; ++k) {
                    const int q = heomk::tile_pos(n, i, k);
                    if (q - i * heomk::tile_stride(n) >= heomk::tile_stride(n) || used[q]++)
                        { printf("bad tile position n=%d (%d,%d)\n", n, i, k); ++bad; }
                }
        }
        // team kernel: conflict-free quarter-warp operand reads (16-byte bank groups: index mod 8)
        // and exchange writes; lanes 8q..8q+7 hold g = 2q, 2q+1 and t = 0..3
        if (n > 8)
            for (int b = 0; b < 2; ++b)
                for (int s = 0; s < 4; ++s)
                    for (int q = 0; q < 4; ++q)
                        for (int which = 0; which < 3; ++which) {
                            int used[8] = {0};
                            for (int g = 2 * q; g <= 2 * q + 1; ++g)
                                for (int t = 0; t < 4; ++t) {
                                    int pos;
                                    if (which == 0) pos = heomk::tile_pos(n, 8 * b + g, 4 * s + t); // A
                                    else if (which == 1) pos = heomk::tile_pos(n, 4 * s + t, 8 * b + g); // B
                                    else pos = (8 * b + g) * heomk::kXchStride + 8 * (s & 1) + 2 * t + (s >> 1); // C: J = s & 1, c0/c1 = s >> 1
                                    if (used[pos % 8]++) { printf("bank conflict n=%d b=%d s=%d q=%d w=%d\n", n, b, s, q, which); ++bad; }
                                }
                        }
    }
    // searched sector tables for N <= 8: coverage, and the bank conflicts of the reads that the kernels make
    for (int n = 1; n <= 8; ++n) {
        const int P = heomk::pairs_of(n);
        int seen[64] = {0};
        for (int p = 0; p < P; ++p) {
            const int e1 = kPairE1[n][p], e2 = kPairE2[n][p];
            if (e1 < 0 || e1 >= n * n || e2 < 0 || e2 >= n * n) { printf("bad table range n=%d\n", n); ++bad; continue; }
            const int i1 = e1 / n, j1 = e1 % n, i2 = e2 / n, j2 = e2 % n;
            const bool d1 = i1 == j1, d2 = i2 == j2;
            if (d1 != d2 || (!d1 && !(i1 == j2 && j1 == i2))) { printf("bad pair n=%d p=%d\n", n, p); ++bad; }
            seen[e1]++;
            if (e2 != e1) seen[e2]++;
        }
        for (int e = 0; e < n * n; ++e)
            if (seen[e] != 1) { printf("bad table coverage n=%d e=%d\n", n, e); ++bad; }
        for (int W = 1; W <= 64; ++W) {
            const int NW = (2 * W + 3) & ~3, TWB = (W + 15) & ~15;
            const int sb = heomk::dmma_slot_bytes(P, NW, TWB), wb = heomk::dmma_warp_bytes(P, NW, TWB);
            if (sb % 16 || wb % 16 || sb < P * 32 + NW * 4 + TWB + 16 + 16 /* zeros */ || wb < 2 * sb + 16) { printf("bad dmma slot n=%d W=%d\n", n, W); ++bad; }
            if (heomk::dmma_smem_bytes(P, W, NW, TWB, 41) > 227 * 1024) { printf("dmma smem too big n=%d W=%d\n", n, W); ++bad; }
        }
    }
    // lockstep order: one more wavefront per quarter warp and slice with all eight lanes inside the tile, the least
    // there is (gen_pair_tables.py); row order: the owner's order leaves less choice (gen_row_tables.py)
    const int lock_extra[9] = {0, 0, 0, 0, 0, 0, 0, 3, 8}, row_extra[9] = {0, 0, 0, 0, 0, 0, 0, 6, 12};
    for (int n = 1; n <= 8; ++n) {
        const int lk = extra_wavefronts(n, kPairE1[n], kPairE2[n], false);
        const int rw = extra_wavefronts(n, kRowE1[n], kRowE2[n], true);
        if (lk > lock_extra[n]) { printf("bank conflicts lockstep n=%d: %d\n", n, lk); ++bad; }
        if (rw > row_extra[n]) { printf("bank conflicts row order n=%d: %d\n", n, rw); ++bad; }
    }
    printf("%s %ld\n", bad ? "FAILED" : "ok", checked);
    return bad ? 1 : 0;
}

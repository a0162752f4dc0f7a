#!/usr/bin/env python3
"""Generate pair_tables.inc: the sector order of the lockstep kernel (N <= 8).

An ADO (N x N complex) is stored as P = N(N-1)/2 + ceil(N/2) sectors of
32 B; each sector holds a symmetric pair (w(i,j), w(j,i)) or two diagonal
elements.  The lockstep kernel computes the commutator of every instance with
FP64 m8n8k4 MMAs on the tile zero-padded to 8 x 8: lane l = 4r + t reads, for
k-slice s, the sector of the pair {r, k}, k = 2t + s, whose two halves are
exactly its A-fragment element (r, k) and its B-fragment element (k, r).

This script searches (simulated annealing) the sector numbering and the
orientation of each pair so that the fragment reads of every quarter warp hit
8 different 16-byte bank groups (no shared-memory bank conflicts).  A diagonal
element is its own transpose: the B fragment reads it where the A fragment
does.  Of a conflict-free A read of eight lanes, the lane that reads the other
half of the same bank groups turns to the diagonal lane's group in the B read,
as all lanes but that one change halves.  So a quarter warp and slice with
all its lanes inside the tile costs at least one wavefront more: N = 8 has
eight of them, N = 7 three, and the search reaches that.  The commutator is
written where the A fragments were read.

Among such orders it looks for one where the sectors of each state's cross (row
and column b) fall into few groups of four neighbours.  A sector of 256
instances is 8 KB, so a cross is read from far apart all the same, yet it shows
(us per stage, 256 instances, depth 6, without / with this rule): 7 states 228.8
/ 225.6, 6 states 100.5 / 101.7; 128 instances of 8 states, depth 5: 99.3 / 99.1.
The result is deterministic for the fixed seeds below.

Usage: python gen_pair_tables.py OUT.inc
"""
import random
import sys
from collections import Counter


def items_of(n):
    off = [(i, j) for i in range(n) for j in range(i + 1, n)]
    diag = [(2 * k, min(2 * k + 1, n - 1)) for k in range((n + 1) // 2)]
    return off, diag


def build(n, perm, orient):
    off, diag = items_of(n)
    table = [None] * len(perm)
    for it, (a, b) in enumerate(off + diag):
        if it < len(off):
            e1, e2 = (a, b), (b, a)
        else:
            e1, e2 = (a, a), (b, b)
        if orient[it] and e1 != e2:
            e1, e2 = e2, e1
        table[perm[it]] = (e1, e2)
    return table


def cost(n, perm, orient):
    """Extra wavefronts of the operand reads of one tile; groups of four sectors that the crosses touch, in hundredths."""
    table = build(n, perm, orient)
    loc = {}
    for sec, (e1, e2) in enumerate(table):
        loc.setdefault(e1, (sec, 0))
        loc.setdefault(e2, (sec, 1))
    c = 0
    for q in range(4):
        for s in range(2):
            for which in (0, 1):
                ch = []
                for rr in (2 * q, 2 * q + 1):
                    for t in range(4):
                        col = 2 * t + s
                        if rr < n and col < n:
                            sec, h = loc[(rr, col) if which == 0 else (col, rr)]
                            ch.append((2 * sec + h) % 8)
                if ch:
                    c += max(Counter(ch).values()) - 1
    groups = sum(len({p // 4 for p, (e1, e2) in enumerate(table) if b in e1 or b in e2}) for b in range(n))
    return c + 0.01 * groups


def search(n, seed):
    off, diag = items_of(n)
    P = len(off) + len(diag)
    rng = random.Random(seed)
    best = None
    for restart in range(8):
        perm = list(range(P))
        rng.shuffle(perm)
        orient = [rng.randint(0, 1) for _ in range(P)]
        cur = cost(n, perm, orient)
        T = 2.0
        for _ in range(30000):
            if rng.random() < 0.6 and P > 1:
                a, b = rng.sample(range(P), 2)
                perm[a], perm[b] = perm[b], perm[a]
                nc = cost(n, perm, orient)
                if nc <= cur or rng.random() < 2.718 ** ((cur - nc) / T):
                    cur = nc
                else:
                    perm[a], perm[b] = perm[b], perm[a]
            else:
                a = rng.randrange(P)
                orient[a] ^= 1
                nc = cost(n, perm, orient)
                if nc <= cur or rng.random() < 2.718 ** ((cur - nc) / T):
                    cur = nc
                else:
                    orient[a] ^= 1
            T = max(0.02, T * 0.9997)
        if best is None or cur < best[0]:
            best = (cur, perm[:], orient[:])
    c, perm, orient = best
    return build(n, perm, orient), c


def main():
    out = sys.argv[1]
    rows = []
    for n in range(1, 9):
        if n == 1:
            table, c = [((0, 0), (0, 0))], 0.01
        else:
            table, c = search(n, 1000 + n)
        e1 = [a[0] * n + a[1] for a, b in table]
        e2 = [b[0] * n + b[1] for a, b in table]
        rows.append((n, e1, e2, c))
        print(f"N={n}: P={len(table)} extra wavefronts={int(c)} groups={round(c % 1 * 100)}", flush=True)
    with open(out, "w") as f:
        f.write("/* Generated by gen_pair_tables.py: sector order of the lockstep kernel (N <= 8).\n"
                " * kPairE1[N][p], kPairE2[N][p] = row-major element index of the two halves of\n"
                " * sector p (equal for the padding half of an odd N's last diagonal sector). */\n")
        f.write("static const signed char kPairE1[9][32] = {\n    {0},\n")
        for n, e1, e2, c in rows:
            f.write("    {" + ", ".join(map(str, e1)) + "}, /* N=%d extra wavefronts=%d groups=%d */\n" % (n, int(c), round(c % 1 * 100)))
        f.write("};\nstatic const signed char kPairE2[9][32] = {\n    {0},\n")
        for n, e1, e2, c in rows:
            f.write("    {" + ", ".join(map(str, e2)) + "},\n")
        f.write("};\n")


if __name__ == "__main__":
    main()
